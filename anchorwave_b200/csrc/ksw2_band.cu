// KSW2 extd2, banded form (w >= 0) and the Singletrack traceback, on sm_100a.
//
// The reference sweeps anti-diagonals r and keeps the int8 difference cells in
// arrays indexed by target position t; on each anti-diagonal it recomputes whole
// SIMD blocks [stB, en16] (st0 rounded down to the block, en0 rounded up to 16),
// so cells just outside the band ("padding") are computed from whatever the arrays
// held, and the in-band cells and the traceback read them
// (minimap2/ksw2_extd2_avx.c:255-701, ksw2_extd2_sse.c:136-331).  This kernel
// computes the same cells in target-column strips swept row by row (the layout of
// the full-matrix kernel) and restates the array semantics cell by cell:
//   * a column's registers hold the last value written at its position, so a
//     column that is not computed on a row keeps its previous values;
//   * left input of cell (t, j): the cell (t-1, j) if it was computed, else the
//     array's initial values; at t == st16 the reference's boundary value
//     (x[st16-1] only on the anti-diagonal where st16 advanced, constants
//     otherwise, the matrix edge when st16 == 0, ksw2_extd2_avx.c:273-287); at
//     t == stB < st16 (lane 0 of the first block) the in-register wrap to lane 15,
//     i.e. cell (stB+15, j-16), kept in a 16-row shared-memory ring;
//   * up input: the column registers, the top-edge values on row 0;
//   * score: the score-fill (ksw2_extd2_avx.c:289-311) refreshes position t on
//     anti-diagonal r when st0 <= t <= st0+16*ceil((en0-st0+1)/16)-1 (en0 for
//     generic scoring); otherwise the stale value of the last fill stays;
//   * H row: H[t] += v[t] inside the band, H[en0] = H[en0-1] + u[en0] on the right
//     edge (ksw2_extd2_sse.c:332-367), mqe/mte with ">=" (:369-372), the score
//     on the last anti-diagonal; the anti-diagonal loop stops at the first empty
//     band (:151-154, zdropped = 1).
// Rows above the matrix (j < 0) only refresh the stale score; rows below it and
// columns right of it never reach a cell of the matrix.
//
// Three forms of a step (one row of every lane), chosen for the whole warp:
//   * interior: every cell strictly inside the band, the full-matrix arithmetic unchanged;
//     the steps where that holds for all lanes are one range of k, solved once per strip;
//   * edge: the rules above from closed forms in the distance of a cell to the band's
//     right edge, e = j + w - t.  The band edge crosses a strip during its first rows and
//     the strip on the right cannot start before, so these steps are the chain that bounds
//     long pairs;
//   * corner (rows 0 and qlen-1, rows above the matrix, and the anti-diagonals where the
//     rule for st0 changes): the same rules from st0 and en0 of every cell.
// The stale scores are kept as the last fill of each column in a register of its own, which
// interior steps refresh for nothing.
//
// Work decomposition: every (pair, strip) is a unit of a device queue, ordered so
// that a strip is always taken after the strip on its left; a warp takes a unit and
// sweeps its rows with the one-row lane skew of the full-matrix kernel, reading its left
// column as the strip on the left writes it.  Many warps, across CTAs, work on one pair at
// once, so a single long interval fills the GPU.  An entry of a boundary column carries a
// mark that says it is written (the columns are cleared before the first pass), so a strip
// reads eight rows ahead and waits (bounded) only for entries that are not there yet: no
// fence and no counter between the strips.
#include "ksw2_band.h"
#include "tb_walk.cuh"

#include <algorithm>
#include <climits>
#include <cstring>

namespace aw {

namespace {

constexpr unsigned FULL = 0xffffffffu;

struct Geom {
    int qlen, tlen, w, nd, rb, bmask;  // bmask = ~(block - 1)
    __device__ __forceinline__ int st0(int r) const { return max(max(0, r - qlen + 1), (r - w + 1) >> 1); }
    __device__ __forceinline__ int en0(int r) const { return min(min(tlen - 1, r), (r + w) >> 1); }
};

__device__ __forceinline__ int prmt_sx(uint32_t lo, uint32_t hi, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
    return (int)r;
}
__device__ __forceinline__ int sx8(uint32_t w) { return (int)(int8_t)(uint8_t)w; }
__device__ __forceinline__ uint32_t pack3(int a, int b, int c, uint32_t top) {
    return (uint32_t)(a & 0xff) | ((uint32_t)(b & 0xff) << 8) | ((uint32_t)(c & 0xff) << 16) | (top << 24);
}
__device__ __forceinline__ int edge_diff(int r, const KswScore &S) {
    return r == 0 ? -S.qe : r < S.long_thres ? -S.e : r == S.long_thres ? S.long_diff : -S.e2;
}

// One cell of the reference recurrence in 32-bit registers (the host routes only
// parameter sets whose int8 intermediates cannot wrap).  xs/vs/x2s: left input in,
// this cell's x/v/x2 out; ut/yt/y2t: up input in, this cell's u/y/y2 out.
template <bool ARGMAX, bool RIGHT>
__device__ __forceinline__ void cell(int s, int &xs, int &vs, int &x2s, int &ut, int &yt, int &y2t, int &d,
                                     const KswScore &S) {
    const int a = xs + vs, b = yt + ut, a2 = x2s + vs, b2 = y2t + ut;
    int z = s;
    if (!ARGMAX) {
        z = __vimax3_s32(z, a, b);
        z = __vimax3_s32(z, a2, b2);
    } else {
        // arg-max by priority tags in the low 4 bits of 16 * candidate: the larger tag wins a
        // tie of values, so the max gives z and the state code at once.  Left-aligned: the
        // first candidate wins a tie (ksw2_extd2_sse.c:244-251), tags s=7 > a=6 > ... > b2=3,
        // code = tag ^ 7; right-aligned: the last (:291-298), tags = codes 0..4.
        constexpr int Ts = RIGHT ? 0 : 7, Ta = RIGHT ? 1 : 6, Tb = RIGHT ? 2 : 5, Ta2 = RIGHT ? 3 : 4,
                      Tb2 = RIGHT ? 4 : 3;
        int zt = __vimax3_s32(s * 16 + Ts, b * 16 + Tb, b2 * 16 + Tb2);
        zt = __vimax3_s32(zt, a * 16 + Ta, a2 * 16 + Ta2);
        d = RIGHT ? (zt & 15) : ((zt & 15) ^ 7);
        z = zt >> 4;
    }
    z = min(z, S.mch);
    const int un = z - vs, vn = z - ut;
    if (!(ARGMAX && RIGHT)) {
        const int nez = -S.e - z, nez2 = -S.e2 - z;
        xs = __viaddmax_s32(a, nez, -S.qe);
        yt = __viaddmax_s32(b, nez, -S.qe);
        x2s = __viaddmax_s32(a2, nez2, -S.qe2);
        y2t = __viaddmax_s32(b2, nez2, -S.qe2);
        if (ARGMAX) {
            d += 0x08 * __viaddmin_s32(xs, S.qe, 1);
            d += 0x10 * __viaddmin_s32(yt, S.qe, 1);
            d += 0x20 * __viaddmin_s32(x2s, S.qe2, 1);
            d += 0x40 * __viaddmin_s32(y2t, S.qe2, 1);
        }
    } else {
        const int aa = a - z + S.q, bb = b - z + S.q, aa2 = a2 - z + S.q2, bb2 = b2 - z + S.q2;
        xs = max(aa, 0) - S.qe;
        yt = max(bb, 0) - S.qe;
        x2s = max(aa2, 0) - S.qe2;
        y2t = max(bb2, 0) - S.qe2;
        d |= (aa >= 0 ? 0x08 : 0) | (bb >= 0 ? 0x10 : 0) | (aa2 >= 0 ? 0x20 : 0) | (bb2 >= 0 ? 0x40 : 0);
    }
    ut = un;
    vs = vn;
}

// The Singletrack tracks (v, u) instead of the state bytes: the Singletrack entries of
// the AVX builds (blocks of 32 or 64 bytes), and ksw_extd2_singletrack_sse (16-byte blocks).
bool singletrack_tracks(int flag, int block) {
    return (flag & AW_EZ_SINGLETRACK) && (block > 16 || (flag & AW_EZ_SSE_SINGLETRACK));
}

__device__ __forceinline__ unsigned long long end_key(int v, int pos) {
    return ((unsigned long long)((uint32_t)v ^ 0x80000000u) << 32) | (uint32_t)pos;
}

__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct BandArgs {
    const uint8_t *qcodes, *tcodes;
    const BandPairDev *pairs;
    const BandStripDev *strips;
    const int2 *units;
    int32_t n_units;
    int32_t *queue, *error;
    uint8_t *tb;
    uint2 *bnd;
    BandRes *res;
    KswScore sc;
    int block, generic;
    // ksw_extd2_singletrack_sse's end rules: strict ">" for mqe/mte (the earliest position
    // wins a tie; minimap2/ksw2_singletrack.cpp:583-586)
    int sse_st;
    int store_ckpt;  // 1: store the traceback of recomputed pairs too (their group passes)
    const unsigned long long *deadline;  // null: no deadline
    // recompute rounds: the pairs' walk states; a round's strips stop at the row the walk has
    // reached (it only moves up and left), strips of a finished walk compute nothing
    const BandWalkState *walk;
};

constexpr uint64_t WAIT_NS = 20ull * 1000 * 1000 * 1000;  // bounded wait on the left strip
// Rows of the left column read at a time: a strip starts a row once the group it lies in is
// written (lane 31 finishes row j 31 steps after lane 0), so a hop between strips costs strip
// width + 31 + PUB lane-steps.
constexpr int PUB = 8;
// Mark of a written boundary entry: the byte above its x, v and x2.
constexpr uint32_t BND_MARK = 0x80000000u;

__device__ __forceinline__ uint2 bnd_load(const uint2 *p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return make_uint2((uint32_t)v, (uint32_t)(v >> 32));
}
__device__ __forceinline__ void bnd_store(uint2 *p, uint32_t x, uint32_t h) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((uint64_t)h << 32 | (x | BND_MARK)) : "memory");
}

// NC target columns per lane (strips of 32*NC columns): 8 for throughput, 4 for a shorter
// pipeline lag between strips when few long pairs run.
template <bool CIGAR, bool RIGHT, bool ST, int NC>
__global__ void __launch_bounds__(256, 2) ksw_band_kernel(BandArgs A) {
    constexpr int C = NC;
    // ARGMAX: the state byte is stored (CIGAR without Singletrack)
    constexpr bool ARGMAX = CIGAR && !ST;
    constexpr int CB = ST ? 2 * C : C;  // traceback bytes per lane-step
    // the block wrap reads column stB+15: lane +D of the stB lane, its last column
    constexpr int D = 16 / C - 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ uint32_t ring[8][16][32];
    const KswScore &S = A.sc;
    const int B = A.block;
    const bool src_lane = B > 16 && lane >= D && (((lane - D) * C) & (B - 1)) == 0;

    for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(A.queue, 1);
        u = __shfl_sync(FULL, u, 0);
        if (u >= A.n_units) break;
        const int2 un = A.units[u];
        const BandPairDev P = A.pairs[un.x];
        const int s = un.y;
        const BandStripDev St = A.strips[P.strip0 + s];
        // the last row this pass needs: the strip's last band row, or in a recompute round the
        // walk's row
        int wlim = INT_MAX;
        if (A.walk) {
            const BandWalkState wk = A.walk[un.x];
            wlim = wk.done ? -1 : wk.j;
        }
        const int jstart = St.jstart, jlo = St.jlo, jend = min(St.jend, wlim);
        if (jend < jlo) continue;  // nothing of this strip is computed
        volatile int32_t *stop_word = &A.res[un.x].stopped;
        if (A.deadline && *stop_word) continue;  // the pair stopped at the deadline
        const Geom g{P.qlen, P.tlen, P.w, P.qlen + P.tlen - 1, P.rb, ~(B - 1)};
        const int qlen = P.qlen, tlen = P.tlen, qm1 = qlen - 1, tm1 = tlen - 1, w = P.w;
        const int rlim = min(g.nd, g.rb);
        const uint8_t *qs = A.qcodes + P.qoff, *ts = A.tcodes + P.toff;
        const int col0 = s * 32 * C + lane * C;
        const bool last_strip = s + 1 == P.nstrip;
        // the strip on the left: its stored rows and, after them, its final H (an empty strip
        // computes nothing, so its column keeps the initial values)
        int prod_lo = 0, prod_hi = -1;
        const uint2 *bnd_prod = nullptr;
        if (s > 0) {
            const BandStripDev Pr = A.strips[P.strip0 + s - 1];
            if (min(Pr.jend, wlim) >= Pr.jlo) {
                prod_lo = Pr.jlo, prod_hi = min(Pr.jend, wlim);
                bnd_prod = A.bnd + Pr.bnd_off;
            }
        }
        // a recompute round reads the columns of the first pass and writes none
        uint2 *bnd_me = lane == 31 && !last_strip && !A.walk ? A.bnd + St.bnd_off : nullptr;
        const bool store_tb = CIGAR && (!P.ckpt || A.store_ckpt);  // this strip's traceback is kept
        // this lane's traceback word of step k: tbp + k * 32 * CB
        uint8_t *tbp = CIGAR ? A.tb + St.tb_off + ((int64_t)(jstart - jlo) * 32 + lane) * CB : nullptr;
        BandRes *R = A.res + un.x;
        // lane constants of the closed-form bounds: floor16 and the block end of the lane's columns
        const int F16 = col0 & ~15, XB = (col0 & g.bmask) + B - 1;
        // Score fill right of the band while st0 = (r-w+1)>>1: en0-st0+1 is w+1 where e is even
        // and w where it is odd, so the fill reaches the columns with e >= -2 pad (even) and
        // e >= 1 - 2 pad (odd), pad = what rounds that length up to 16.
        const int fill_even = A.generic ? 0 : 2 * (-(w + 1) & 15), fill_odd = A.generic ? -1 : 2 * (-w & 15) - 1;
        // rows where the lane's cells all lie strictly inside the band, with natural neighbours
        const int fa = max(1, col0 + C + 1 - w);
        const int fb = col0 + C > tm1 ? -1 : min(min(qlen - 2, rlim - col0 - C), col0 > 0 ? col0 + w - 2 : w);
        // steps where that holds for every lane
        const int kf0 = (int)__reduce_max_sync(FULL, max(fa, jstart) + lane) - jstart;
        const int kf1 = (int)__reduce_min_sync(FULL, min(fb, jend) + lane) - jstart + 1;

        int ut[C], yt[C], y2t[C], H[C], ss[C];
        uint32_t rlo[C], rhi[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int t = col0 + c;
            const int tc = t < tlen ? (ts[t] & 7) : 0;
            rlo[c] = S.tab_lo[tc];
            rhi[c] = S.tab_hi[tc];
            ut[c] = -S.qe, yt[c] = -S.qe, y2t[c] = -S.qe2;
            H[c] = AW_NEG_INF;
            ss[c] = 0;
        }
        const uint32_t init_pack = pack3(-S.qe, -S.qe, -S.qe2, 0);
        uint32_t carry = 0;
        int Hcarry = AW_NEG_INF;
        unsigned long long mte_key = 0;  // last strip: the lane that owns the last column
        const int pm = A.sse_st ? INT_MAX : 0;  // strict end rule: mirrored positions
        // lane 0's left values of row jr: x, v, x2 with the mark, and the H on the left
        auto left_of = [&](int jr) -> uint2 {
            if (s == 0) return make_uint2(pack3(-S.qe, edge_diff(jr, S), -S.qe2, 0) | BND_MARK, (uint32_t)AW_NEG_INF);
            if (!bnd_prod || jr < prod_lo) return make_uint2(init_pack | BND_MARK, (uint32_t)AW_NEG_INF);
            return bnd_load(bnd_prod + (min(jr, prod_hi + 1) - prod_lo));
        };
        auto code_of = [&](int jr) -> uint32_t { return jr >= 0 && jr < qlen ? qs[jr] : 0u; };
        // lane i holds what lane 0 needs for row jstart + (k & ~31) + i: the next group's entries
        // and the next 32 query codes are on their way while the current ones are used
        uint2 ahead = make_uint2(BND_MARK, 0u);
        if (lane < PUB) ahead = left_of(jstart + lane);
        uint32_t qnext = code_of(jstart + lane), qcur = 0, bx = 0;
        int bh = 0;
        bool failed = false, stopped = false;
        const int nsteps = jend - jstart + 32;
        for (int kb = 0; kb < nsteps; kb += PUB) {
            if ((kb & 31) == 0) {
                if (A.deadline) {
                    // cooperative stop, polled every 32 rows (ksw2_progress.c:30-38 polls every
                    // 256 anti-diagonals); the pair's other strips see the flag and stop too
                    int st = 0;
                    if (lane == 0) {
                        st = *stop_word;
                        if (!st && aw_deadline_passed(A.deadline)) st = 1, atomicExch((int32_t *)stop_word, 1);
                    }
                    if (__shfl_sync(FULL, st, 0)) {
                        stopped = true;
                        break;
                    }
                }
                qcur = qnext;
                qnext = code_of(jstart + kb + 32 + lane);
            }
            const bool mine = (lane & ~(PUB - 1)) == (kb & 31);
            if (!__all_sync(FULL, !mine || (ahead.x & BND_MARK))) {
                // the left strip is not there yet: poll with back-off; the bound and the error
                // flag (another warp gave up) are checked every 32 polls
                const uint64_t t0 = globaltimer();
                unsigned ns = 16, polls = 0;
                for (;;) {
                    if (mine && !(ahead.x & BND_MARK)) ahead = left_of(jstart + (kb & ~31) + lane);
                    if (__all_sync(FULL, !mine || (ahead.x & BND_MARK))) break;
                    if (A.deadline && __shfl_sync(FULL, lane == 0 ? *stop_word : 0, 0)) {
                        stopped = true;  // the left strip stopped
                        break;
                    }
                    if ((++polls & 31) == 0) {
                        const int bad = globaltimer() - t0 > WAIT_NS || *(volatile int32_t *)A.error;
                        if (__any_sync(FULL, bad)) {
                            failed = true;
                            break;
                        }
                    }
                    __nanosleep(ns);
                    ns = ns < 256 ? ns * 2 : ns;
                }
                if (failed && lane == 0) atomicExch(A.error, 1);
                if (failed || stopped) break;
            }
            if (mine) bx = (ahead.x & 0xffffffu) | qcur << 24, bh = (int)ahead.y;
            if ((lane & ~(PUB - 1)) == ((kb + PUB) & 31)) ahead = left_of(jstart + ((kb + PUB) & ~31) + lane);
            const int kend = min(kb + PUB, nsteps);
            int k = kb;
            if (k >= kf0 && kend <= kf1) {
                // interior: no tests inside the group
#pragma unroll 1
                for (; k < kend; ++k) {
                    uint32_t in = __shfl_up_sync(FULL, carry, 1);
                    const uint32_t b = __shfl_sync(FULL, bx, k & 31);
                    if (lane == 0) in = b;
                    int xs = sx8(in), vs = sx8(in >> 8), x2s = sx8(in >> 16);
                    const uint32_t qc = in >> 24, sel = qc * 0x1111u + 0x8880u;
                    uint32_t w0 = 0, w1 = 0, w2 = 0, w3 = 0;
                    if (ARGMAX && !store_tb) {
                        // no traceback is kept for this strip (a recomputed pair's first pass, or a
                        // pair whose band empties): the cells without their state bytes
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            int d = 0;
                            ss[c] = prmt_sx(rlo[c], rhi[c], sel);
                            cell<false, RIGHT>(ss[c], xs, vs, x2s, ut[c], yt[c], y2t[c], d, S);
                            H[c] += vs;
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            int d = 0;
                            ss[c] = prmt_sx(rlo[c], rhi[c], sel);
                            cell<ARGMAX, RIGHT>(ss[c], xs, vs, x2s, ut[c], yt[c], y2t[c], d, S);
                            H[c] += vs;
                            if (ARGMAX) {
                                if (c < 4) w0 |= (uint32_t)d << (8 * c);
                                else w1 |= (uint32_t)d << (8 * (c - 4));
                            } else if (ST) {
                                if (c < 4) w0 |= (uint32_t)(vs & 0xff) << (8 * c), w2 |= (uint32_t)(ut[c] & 0xff) << (8 * c);
                                else w1 |= (uint32_t)(vs & 0xff) << (8 * (c - 4)), w3 |= (uint32_t)(ut[c] & 0xff) << (8 * (c - 4));
                            }
                        }
                        if (store_tb) {
                            uint8_t *dst = tbp + (int64_t)k * (32 * CB);
                            if (C == 8) {
                                if (ST) __stcs(reinterpret_cast<uint4 *>(dst), make_uint4(w0, w1, w2, w3));
                                else __stcs(reinterpret_cast<uint2 *>(dst), make_uint2(w0, w1));
                            } else {
                                if (ST) __stcs(reinterpret_cast<uint2 *>(dst), make_uint2(w0, w2));
                                else __stcs(reinterpret_cast<uint32_t *>(dst), w0);
                            }
                        }
                    }
                    carry = pack3(xs, vs, x2s, qc);
                    Hcarry = H[C - 1];
                    if (src_lane && k >= kf1 - 16) ring[warp][k & 15][lane] = carry;  // the wrap looks 16 rows back
                    if (bnd_me) bnd_store(bnd_me + (jstart + k - 31 - jlo), carry & 0xffffffu, (uint32_t)Hcarry);
                }
                __syncwarp();
                continue;
            }
#pragma unroll 1
            for (; k < kend; ++k) {
                uint32_t in = __shfl_up_sync(FULL, carry, 1);
                int Hl = __shfl_up_sync(FULL, Hcarry, 1);
                const uint32_t b = __shfl_sync(FULL, bx, k & 31);
                const int hb = __shfl_sync(FULL, bh, k & 31);
                if (lane == 0) in = b, Hl = hb;
                const int j = jstart + k - lane, r0 = col0 + j;
                int xs = sx8(in), vs = sx8(in >> 8), x2s = sx8(in >> 16);
                const uint32_t qc = in >> 24, sel = (j < 0 ? 0u : qc) * 0x1111u + 0x8880u;
                const bool active = j >= jstart && j <= jend;
                // Closed forms of the per-cell geometry over this lane-step (cell c: t = col0+c,
                // r = r0+c, e = e0-c): in band <=> cB <= c <= cE; computed (stB <= t <= en16) <=>
                // cRlo <= c <= cRhi; score filled <=> cB <= c <= fill0 (even c), fill1 (odd c).
                const int e0 = j + w - col0, cB = j - w - col0;
                const int cmax = min(tm1 - col0, rlim - 1 - r0), cE = min(e0, cmax);
                const int cRlo = 2 * (F16 - col0) - cB - 2 * w;
                const int cRhi = min(min(XB + qm1, 2 * XB + w) - r0, cmax);
                // the rule for st0: r-qlen+1 once it is above (r-w+1)>>1, where the fill's length
                // rounds up with the rows left below
                const bool tail0 = r0 - qm1 > ((r0 - w + 1) >> 1), tail1 = r0 + C - 1 - qm1 > ((r0 + C - w) >> 1);
                const bool corner = active && (j < 1 || j >= qm1 || (tail0 != tail1 && cRhi > cE));
                uint32_t w0 = 0, w1 = 0, w2 = 0, w3 = 0;  // traceback bytes of this lane-step
                if (!__any_sync(FULL, corner)) {
                    if (active) {
                        const int f = tail0 ? (A.generic ? 0 : 2 * ((qm1 - j) & 15)) : 0;
                        const bool odd = e0 & 1;
                        const int fill0 = e0 + (tail0 ? f : odd ? fill_odd : fill_even);
                        const int fill1 = e0 + (tail0 ? f : odd ? fill_even : fill_odd);
                        // the band-edge lane st16 and the block wrap stB can only be column col0 (c = 0)
                        if (r0 < rlim) {
                            const int st0 = g.st0(r0), st16 = st0 & ~15, stB = st0 & g.bmask;
                            if (col0 == st16) {
                                if (st16 == 0) xs = -S.qe, vs = edge_diff(j, S), x2s = -S.qe2;
                                else if ((g.st0(r0 - 1) & ~15) == st16) xs = -S.qe, vs = -S.qe, x2s = -S.qe2;
                            } else if (col0 == stB) {
                                const uint32_t wv = ring[warp][(k + D) & 15][lane + D];
                                xs = sx8(wv), vs = sx8(wv >> 8), x2s = sx8(wv >> 16);
                            }
                        }
                        const int ctm = tm1 - col0;
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            const bool inBand = c >= cB && c <= cE;
                            const bool inR = c >= cRlo && c <= cRhi;
                            const bool fresh = c >= cB && c <= ((c & 1) ? fill1 : fill0);
                            const int sc = prmt_sx(rlo[c], rhi[c], sel);
                            ss[c] = fresh ? sc : ss[c];
                            int uu = ut[c], yy = yt[c], yy2 = y2t[c], d = 0;
                            cell<ARGMAX, RIGHT>(ss[c], xs, vs, x2s, uu, yy, yy2, d, S);
                            // H[en0] = H[en0-1] + u on the right edge of the band, else H += v
                            const bool re = (c >= e0 - 1 || c == ctm) && (c > 0 || col0 > 0);
                            const int hn = re ? Hl + uu : H[c] + vs;
                            H[c] = inBand ? hn : H[c];
                            Hl = H[c];
                            ut[c] = inR ? uu : ut[c], yt[c] = inR ? yy : yt[c], y2t[c] = inR ? yy2 : y2t[c];
                            if (ARGMAX) {
                                const uint32_t dd = inR ? (uint32_t)d : 0u;
                                if (c < 4) w0 |= dd << (8 * c);
                                else w1 |= dd << (8 * (c - 4));
                            } else if (ST) {
                                const uint32_t bv = inR ? (uint32_t)(vs & 0xff) : 0u, bu = inR ? (uint32_t)(uu & 0xff) : 0u;
                                if (c < 4) w0 |= bv << (8 * c), w2 |= bu << (8 * c);
                                else w1 |= bv << (8 * (c - 4)), w3 |= bu << (8 * (c - 4));
                            }
                            xs = inR ? xs : -S.qe, vs = inR ? vs : -S.qe, x2s = inR ? x2s : -S.qe2;
                        }
                        if (last_strip) {
                            // H of the last column in band: the largest, later rows on a tie
#pragma unroll
                            for (int c = 0; c < C; ++c)
                                if (c == ctm && c >= cB && c <= cE) {
                                    const unsigned long long key = end_key(H[c], pm ^ j);
                                    mte_key = key > mte_key ? key : mte_key;
                                }
                        }
                        carry = pack3(xs, vs, x2s, qc);
                        Hcarry = Hl;
                    }
                } else if (active) {
                    int fx = xs, fv = vs, fx2 = x2s, Hf = Hl;
                    if (r0 < rlim && j >= 0) {
                        const int st0 = g.st0(r0), st16 = st0 & ~15, stB = st0 & g.bmask;
                        if (col0 == st16) {
                            if (st16 == 0) fx = -S.qe, fv = edge_diff(j, S), fx2 = -S.qe2;
                            else if ((g.st0(r0 - 1) & ~15) == st16) fx = -S.qe, fv = -S.qe, fx2 = -S.qe2;
                        } else if (col0 == stB) {
                            const uint32_t wv = ring[warp][(k + D) & 15][lane + D];
                            fx = sx8(wv), fv = sx8(wv >> 8), fx2 = sx8(wv >> 16);
                        }
                    }
                    const bool top = j == 0;
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const int t = col0 + c, r = r0 + c;
                        if (t <= tm1 && r >= 0 && r < rlim) {
                            const int st0 = g.st0(r), en0 = g.en0(r);
                            const int fe = A.generic ? en0 : st0 + ((en0 - st0 + 16) & ~15) - 1;
                            if (st0 <= t && t <= fe) ss[c] = prmt_sx(rlo[c], rhi[c], sel);
                        }
                        if (j < 0) continue;  // above the matrix: only the score fill of the reference runs here
                        const bool inBand = c >= cB && c <= cE;
                        const bool inR = c >= cRlo && c <= cRhi;
                        int lx = fx, lv = fv, lx2 = fx2;
                        int uu = top ? edge_diff(t, S) : ut[c];
                        int yy = top ? -S.qe : yt[c], yy2 = top ? -S.qe2 : y2t[c];
                        int d = 0;
                        cell<ARGMAX, RIGHT>(ss[c], lx, lv, lx2, uu, yy, yy2, d, S);
                        if (inR) ut[c] = uu, yt[c] = yy, y2t[c] = yy2;
                        fx = inR ? lx : -S.qe, fv = inR ? lv : -S.qe, fx2 = inR ? lx2 : -S.qe2;
                        const bool re = t == tm1 || top || c >= e0 - 1;
                        const int hn = r == 0 ? lv - S.qe_pre : (re && t > 0) ? Hf + uu : H[c] + lv;
                        if (inBand) {
                            H[c] = hn;
                            // end tracking straight into the pair's record (rare cells; the
                            // packed keys make the ">=" later-wins rule an unsigned max, and
                            // the strict earlier-wins rule one on the mirrored position)
                            if (re && t == tm1) atomicMax(&R->mte_key, end_key(hn, pm ^ j));
                            if (j == qm1) atomicMax(&R->mqe_key, end_key(hn, pm ^ t));
                            if (j == qm1 && t == tm1) R->score = hn, R->has_score = 1;
                        }
                        if (ARGMAX) {
                            const uint32_t dd = inR ? (uint32_t)d : 0u;
                            if (c < 4) w0 |= dd << (8 * c);
                            else w1 |= dd << (8 * (c - 4));
                        } else if (ST) {
                            const uint32_t bv = inR ? (uint32_t)(lv & 0xff) : 0u, bu = inR ? (uint32_t)(uu & 0xff) : 0u;
                            if (c < 4) w0 |= bv << (8 * c), w2 |= bu << (8 * c);
                            else w1 |= bv << (8 * (c - 4)), w3 |= bu << (8 * (c - 4));
                        }
                        Hf = H[c];
                    }
                    if (j < 0) fx = -S.qe, fv = -S.qe, fx2 = -S.qe2, Hf = H[C - 1];
                    carry = pack3(fx, fv, fx2, qc);
                    Hcarry = Hf;
                }
                if (active) {
                    if (src_lane) ring[warp][k & 15][lane] = carry;
                    if (j >= jlo) {
                        if (store_tb) {
                            uint8_t *dst = tbp + (int64_t)k * (32 * CB);
                            if (C == 8) {
                                if (ST) __stcs(reinterpret_cast<uint4 *>(dst), make_uint4(w0, w1, w2, w3));
                                else __stcs(reinterpret_cast<uint2 *>(dst), make_uint2(w0, w1));
                            } else {
                                if (ST) __stcs(reinterpret_cast<uint2 *>(dst), make_uint2(w0, w2));
                                else __stcs(reinterpret_cast<uint32_t *>(dst), w0);
                            }
                        }
                        if (bnd_me) bnd_store(bnd_me + (j - jlo), carry & 0xffffffu, (uint32_t)Hcarry);
                    }
                }
                if (B > 16) __syncwarp();
            }
        }
        if (failed) break;
        if (stopped) continue;
        // the strip's final H, for the rows below its last one
        if (bnd_me) bnd_store(bnd_me + (jend - jlo + 1), init_pack, (uint32_t)Hcarry);
        if (mte_key) atomicMax(&R->mte_key, mte_key);
    }
}

// ---- traceback --------------------------------------------------------------------

struct BtArgs {
    const BandPairDev *pairs;
    int npair;
    const BandStripDev *strips;
    const uint8_t *tb;
    const BandRes *res;
    BandWalkState *walk;
    const uint8_t *qcodes, *tcodes;
    KswOut *out;
    uint32_t *cig;
    KswScore sc;
    int8_t mat[64];
    int m, flag, block;
};

// The move that ksw_backtrack's off/off_end forcing takes outside the computed blocks of the
// cell's anti-diagonal (1: deletion, 2: insertion), or -1.
__device__ __forceinline__ int band_force(const Geom &g, int i, int j) {
    const int r = i + j;
    return i > (g.en0(r) | 15) ? 1 : i < (g.st0(r) & g.bmask) ? 2 : -1;
}

// The stored rows of a column group of a pair's strips (words of WB bytes).
template <int WB, int NC>
__device__ __forceinline__ TbGroup band_group(const BandStripDev *strips, const uint8_t *tb, int tlen, int col_lo,
                                              int gg) {
    if (gg < 0 || gg * NC >= tlen || gg * NC < col_lo) return TbGroup{tb, 0, -1};
    const BandStripDev St = strips[gg >> 5];
    const int L = gg & 31;
    return TbGroup{tb + St.tb_off + ((int64_t)L * 32 + L) * WB, St.jlo, St.jend};
}

// Warps per block of the finishing kernel: the Singletrack words are twice as large, and its
// gap search has two tiles of its own.
template <bool ST>
constexpr int fin_warps() { return ST ? 1 : 4; }

// Result record of one pair, then ksw_backtrack (minimap2/ksw2.h:160-192) with the
// off/off_end forcing of the band, or the Singletrack reconstruction
// (minimap2/ksw2_singletrack.cpp:63-176); one warp per pair walks in runs (tb_walk.cuh).
template <bool ST, int NC>
__global__ void __launch_bounds__(32 * fin_warps<ST>()) ksw_band_finish_kernel(BtArgs A) {
    constexpr int WB = ST ? 2 * NC : NC;  // bytes per lane-word: NC columns (v then u for Singletrack)
    using Window = TbWindow<WB, NC, ST ? 1 : 0, true>;
    using Probe = TbWindow<WB, NC, 0, false>;  // the rows and columns of a Singletrack gap search
    __shared__ __align__(16) uint8_t tiles[fin_warps<ST>()][Window::BYTES + (ST ? Probe::BYTES : 0)];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pi = blockIdx.x * fin_warps<ST>() + warp;
    if (pi >= A.npair) return;
    const BandPairDev P = A.pairs[pi];
    const BandRes R = A.res[pi];
    const Geom g{P.qlen, P.tlen, P.w, P.qlen + P.tlen - 1, P.rb, ~(A.block - 1)};
    const int qlen = P.qlen, tlen = P.tlen, flag = A.flag;
    KswOut o;
    o.max = 0, o.max_q = -1, o.max_t = -1, o.reach_end = 0, o.stopped = 0, o.n_cigar = 0;
    o.score = R.has_score ? R.score : AW_NEG_INF;
    o.mqe = R.mqe_key ? (int)((uint32_t)(R.mqe_key >> 32) ^ 0x80000000u) : AW_NEG_INF;
    // ksw_extd2_singletrack_sse: positions stored mirrored (its strict ">"), and
    // mte_q = r - en with en rounded up to its 16-byte block (minimap2/ksw2_singletrack.cpp:583-586)
    const bool sse_st = (flag & AW_EZ_SINGLETRACK) && (flag & AW_EZ_SSE_SINGLETRACK);
    const int pm = sse_st ? INT_MAX : 0;
    o.mqe_t = R.mqe_key ? pm ^ (int)(uint32_t)R.mqe_key : -1;
    o.mte = R.mte_key ? (int)((uint32_t)(R.mte_key >> 32) ^ 0x80000000u) : AW_NEG_INF;
    o.mte_q = R.mte_key ? (pm ^ (int)(uint32_t)R.mte_key) - (sse_st ? ((tlen + 15) & ~15) - tlen : 0) : -1;
    o.zdropped = P.rb < g.nd ? 1 : 0;
    if (R.stopped) {
        // stopped at the deadline: no score and no traceback (ksw2_extd2_sse.c:136-139, :400-409)
        o.stopped = 1, o.score = AW_NEG_INF;
        if (lane == 0) {
            if (P.ckpt) A.walk[pi].done = 1;
            A.out[P.idx] = o;
        }
        return;
    }
    const bool cigar = !(flag & AW_EZ_SCORE_ONLY);
    const BandStripDev *strips = A.strips + P.strip0;
    const uint8_t *tb = A.tb;
    Window win;
    win.init(tiles[warp], 32 * WB);
    auto grp = [&](int gg) -> TbGroup { return band_group<WB, NC>(strips, tb, tlen, 0, gg); };
    WarpCigar cg{A.cig + P.cig_off, 0, 0, 0};
    if (cigar && ST) {
        // ksw_extd2_singletrack_sse reconstructs whatever the EXTZ/SEMIGLOBAL flags
        // (minimap2/ksw2_singletrack.cpp:606-615)
        if (!o.zdropped && (sse_st || !(flag & (AW_EZ_EXTZ_ONLY | AW_EZ_SEMIGLOBAL_END)))) {
            const uint8_t *qs = A.qcodes + P.qoff, *ts = A.tcodes + P.toff;
            Probe probe;
            probe.init(tiles[warp] + Window::BYTES, 32 * WB);
            int i = tlen - 1, j = qlen - 1;
            if (tb_singletrack(i, j, cg, win, probe, grp, [&](int a, int c) { return band_force(g, a, c); }, A.sc, A.mat,
                               A.m, qs, ts)) {
                if (i >= 0) cg.push(2, i + 1);
                if (j >= 0) cg.push(1, j + 1);
                o.n_cigar = cg.finish(true);
            }
            if (o.n_cigar == 0) o.zdropped = 1;
        } else if (!o.zdropped) {
            o.zdropped = 1;
        }
    } else if (cigar) {
        int i0 = -1, j0 = -1;
        if (!o.zdropped && (flag & AW_EZ_SEMIGLOBAL_END)) {
            if (o.mqe > o.mte) o.score = o.mqe, i0 = o.mqe_t, j0 = qlen - 1;
            else o.score = o.mte, i0 = tlen - 1, j0 = o.mte_q;
        } else if (!o.zdropped && !(flag & AW_EZ_EXTZ_ONLY)) {
            i0 = tlen - 1, j0 = qlen - 1;
        }
        if (P.ckpt) {
            // traceback recomputed group by group (ksw_band_walk_kernel); start state only
            if (lane == 0) {
                BandWalkState w;
                w.i = i0, w.j = j0, w.state = 0, w.n = 0, w.op = 0, w.len = 0, w.pad = 0;
                w.done = (i0 >= 0 || j0 >= 0) ? 0 : 1;
                A.walk[pi] = w;
            }
        } else if (i0 >= 0 || j0 >= 0) {
            int i = i0, j = j0, state = 0;
            tb_walk(i, j, state, 0, cg, win, grp, [&](int a, int b) { return band_force(g, a, b); });
            if (i >= 0) cg.push(2, i + 1);
            if (j >= 0) cg.push(1, j + 1);
            o.n_cigar = cg.finish(!(flag & AW_EZ_REV_CIGAR));
        }
    }
    if (lane == 0) A.out[P.idx] = o;
}

// One group of a recomputed pair per block (a round's groups): continue the ksw_backtrack
// walk through the group's freshly stored traceback until it leaves the group on the left
// (or ends); in the pair's first group, close the walk (the leading gap, the reversal, the
// CIGAR length).
template <int NC>
__global__ void __launch_bounds__(32) ksw_band_round_walk_kernel(BtArgs A, const BandGroupDev *groups) {
    using Window = TbWindow<NC, NC, 0, true>;
    __shared__ __align__(16) uint8_t tiles[Window::BYTES];
    const BandGroupDev G = groups[blockIdx.x];
    const int slot = G.slot, col_lo = G.col_lo;
    BandWalkState w = A.walk[slot];
    if (w.done) return;
    const BandPairDev P = A.pairs[slot];
    if (A.res[slot].stopped) {
        // the group's recomputation stopped at the deadline: its traceback is incomplete
        if ((threadIdx.x & 31) == 0) {
            A.walk[slot].done = 1;
            A.out[P.idx].stopped = 1, A.out[P.idx].score = AW_NEG_INF, A.out[P.idx].n_cigar = 0;
        }
        return;
    }
    const Geom g{P.qlen, P.tlen, P.w, P.qlen + P.tlen - 1, P.rb, ~(A.block - 1)};
    const int tlen = P.tlen;
    const BandStripDev *strips = A.strips + P.strip0;
    const uint8_t *tb = A.tb;
    Window win;
    win.init(tiles, 32 * NC);
    auto grp = [&](int gg) -> TbGroup { return band_group<NC, NC>(strips, tb, tlen, col_lo, gg); };
    WarpCigar cg{A.cig + P.cig_off, w.n, (uint32_t)w.op, w.len};
    int i = w.i, j = w.j, state = w.state;
    tb_walk(i, j, state, col_lo, cg, win, grp, [&](int a, int b) { return band_force(g, a, b); });
    if (G.last) {
        if (i >= 0) cg.push(2, i + 1);
        if (j >= 0) cg.push(1, j + 1);
        const int n = cg.finish(!(A.flag & AW_EZ_REV_CIGAR));
        if ((threadIdx.x & 31) == 0) {
            A.out[P.idx].n_cigar = n;
            A.walk[slot].done = 1;
        }
        return;
    }
    if ((threadIdx.x & 31) == 0) {
        w.i = i, w.j = j, w.state = state, w.n = cg.n, w.op = (int)cg.op, w.len = cg.len;
        A.walk[slot] = w;
    }
}

template <bool CIGAR, bool RIGHT, bool ST>
void *kernel_ptr() {
    return (void *)ksw_band_kernel<CIGAR, RIGHT, ST, 8>;
}

void *band_kernel_for(int flag, int block) {
    const bool cigar = !(flag & AW_EZ_SCORE_ONLY), right = !!(flag & AW_EZ_RIGHT);
    const bool st = cigar && singletrack_tracks(flag, block);
    if (st) return kernel_ptr<true, false, true>();
    if (cigar && right) return kernel_ptr<true, true, false>();
    if (cigar) return kernel_ptr<true, false, false>();
    return kernel_ptr<false, false, false>();
}

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Device bytes of a pair's boundary columns (entries rounded as the wave packs them).
int64_t band_bnd_bytes(int64_t entries) { return (entries + 31) / 32 * 32 * (int64_t)sizeof(uint2); }

}  // namespace

int band_break(int qlen, int tlen, int w) {
    const int nd = qlen + tlen - 1;
    int rb = nd;
    if (w == 0 && nd > 1) rb = 1;
    // both conditions below are monotone in r (ksw2_extd2_sse.c:147-154: st > en)
    int lo = 0, hi = nd;
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2;
        if (mid - qlen + 1 > ((mid + w) >> 1)) hi = mid;
        else lo = mid + 1;
    }
    rb = std::min(rb, lo);
    lo = 0, hi = nd;
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2;
        if (((mid - w + 1) >> 1) > tlen - 1) hi = mid;
        else lo = mid + 1;
    }
    return std::min(rb, lo);
}

int64_t band_cells(int qlen, int tlen, int w) {
    if (w < 0) w = std::max(qlen, tlen);
    const int rb = band_break(qlen, tlen, w);
    int64_t total = 0;
    for (int r = 0; r < rb; ++r) {
        const int st = std::max(std::max(0, r - qlen + 1), (r - w + 1) >> 1);
        const int en = std::min(std::min(tlen - 1, r), (r + w) >> 1);
        total += en - st + 1;
    }
    return total;
}

int band_plan_build(BandPlan &bp, const std::vector<int32_t> &ids, const std::vector<int> &qlen,
                    const std::vector<int> &tlen, const std::vector<int> &w, const std::vector<KswPair> &pairs,
                    int flag, int block, int64_t tb_budget, int nc, std::vector<int32_t> *refused) {
    bp = BandPlan();
    bp.block = block;
    bp.nc = nc == 4 ? 4 : 8;
    const int SW = 32 * bp.nc;  // strip width
    const bool cigar = !(flag & AW_EZ_SCORE_ONLY);
    const bool st = cigar && singletrack_tracks(flag, block);
    const int CB = st ? 2 * bp.nc : bp.nc;  // traceback bytes per lane-step
    const int B = block;
    struct PairGeo {
        int32_t id, ww, rb;
        int64_t tb, bnd;
        bool ckpt = false, refused = false, notb = false;
        std::vector<BandStripDev> strips;
        std::vector<int64_t> start;  // estimated start step of each strip
        std::vector<int64_t> stb;    // traceback bytes of each strip
    };
    std::vector<PairGeo> geo(ids.size());
    for (size_t a = 0; a < ids.size(); ++a) {
        PairGeo &G = geo[a];
        const int i = ids[a], ql = qlen[i], tl = tlen[i];
        const int ww = w[i] < 0 ? std::max(ql, tl) : std::min(w[i], std::max(ql, tl));
        G.id = i, G.ww = ww, G.rb = band_break(ql, tl, ww);
        const int nd = ql + tl - 1;
        const int nstrip = (int)ceil_div(tl, SW);
        G.tb = 0, G.bnd = 0;
        int64_t T = 0;
        int prev_js = 0;
        for (int s = 0; s < nstrip; ++s) {
            const int c0 = s * SW;
            BandStripDev sd;
            // rows the strip sweeps: from the first score-fill row of any of its columns
            // (fills reach 15 past en0, so no earlier than c0-w-31, and no row above -15)
            // to the last row where one of its columns is computed (stB <= t)
            sd.jstart = (int)std::max<int64_t>(-15, (int64_t)c0 - ww - 32);
            sd.jlo = std::max(0, sd.jstart);
            int64_t jend = -1;
            for (int tg = c0; tg < std::min(c0 + SW, tl); tg += B) {
                const int64_t X = (int64_t)tg + B - 1;
                const int64_t b = std::min<int64_t>(std::min<int64_t>(nd - 1, (int64_t)G.rb - 1),
                                                    std::min<int64_t>(X + ql - 1, 2 * X + ww));
                jend = std::max(jend, b - tg);
            }
            sd.jend = (int)std::min<int64_t>(jend, ql - 1);
            const int64_t rows = sd.jend >= sd.jlo ? (int64_t)sd.jend - sd.jlo + 1 : 0;
            sd.tb_off = G.tb;  // relative to the pair until the wave is packed
            sd.bnd_off = G.bnd;
            int64_t stb = 0;
            if (rows > 0) {
                if (cigar) stb = (rows + 31) * 32 * CB;
                G.tb += stb;
                G.bnd += rows + 1;
            }
            G.stb.push_back(stb);
            // estimated start: the left strip must have swept this strip's first rows
            T += (s == 0 ? 0 : std::max(0, sd.jstart - prev_js) + 64);
            prev_js = sd.jstart;
            G.strips.push_back(sd);
            G.start.push_back(T);
        }
        G.tb = (G.tb + 255) / 256 * 256;
        if (G.rb < nd) {
            // the band becomes empty before the end: the reference stops there with
            // zdropped = 1 and no traceback (ksw2_extd2_sse.c:151-154), so the DP runs without
            // storing one (the first pass of a recomputed pair, with nothing to recompute)
            G.ckpt = G.notb = true;
            G.tb = 0;
        }
    }
    // The budget is split once between the boundary-column arena and the traceback arena
    // (both are sized for their largest wave): the boundary columns get what the whole batch
    // needs, up to a third of the budget; the traceback arena the rest.  A wave's boundary
    // columns and its tracebacks stored in full must fit their arenas; the recompute rounds of
    // its recomputed pairs use the whole traceback arena after the wave's other walks.
    int64_t bnd_all = 0;
    for (const PairGeo &G : geo) bnd_all += band_bnd_bytes(G.bnd);
    const int64_t cap_bnd = std::min(bnd_all, tb_budget / 3);
    const int64_t cap_tb = std::max<int64_t>(tb_budget - cap_bnd, 1);
    const int64_t gres = cap_tb;
    for (PairGeo &G : geo) {
        if (G.notb) continue;
        // Singletrack pairs keep their whole two-track traceback: the reconstruction probes
        // arbitrarily far left in one gap search, so it cannot be split into strip groups.  A
        // pair whose traceback does not fit is refused like an allocation failure of the
        // reference (ksw2_extd2_avx.c:206-210: reset result, zdropped = 1).
        bool refuse = st && G.tb > cap_tb;
        if (!st && G.tb > cap_tb) {
            // Traceback beyond the budget: the first pass stores only the strips' boundary
            // columns; then the traceback is recomputed in groups of strips, from the last group
            // to the first, each from the stored column on its left, and the walk continues
            // through each group as it is recomputed.  The groups are cut per wave (below).
            for (int s = 0; s < (int)G.strips.size(); ++s) refuse |= G.stb[s] > cap_tb;
            if (!refuse) {
                G.ckpt = true;
                G.tb = 0;  // the first pass stores no traceback
            }
        }
        if (refuse) {
            if (!refused) return AW_E_NOMEM_INTERNAL;
            G.refused = true;
            refused->push_back(G.id);
        }
    }
    for (const PairGeo &G : geo) {
        if (G.refused) continue;
        bp.tb_total += G.tb;
        bp.cells += band_cells(qlen[G.id], tlen[G.id], G.ww);
    }
    // Pairs largest first into the fewest waves whose boundary columns and tracebacks stored in
    // full fit their arenas (LPT multiway fit), or one pair alone.
    std::vector<size_t> ord;
    for (size_t a = 0; a < ids.size(); ++a)
        if (!geo[a].refused) ord.push_back(a);
    std::sort(ord.begin(), ord.end(), [&](size_t x, size_t y) {
        const int64_t cx = (int64_t)qlen[geo[x].id] * geo[x].ww, cy = (int64_t)qlen[geo[y].id] * geo[y].ww;
        return cx != cy ? cx > cy : geo[x].id < geo[y].id;
    });
    std::vector<std::vector<size_t>> wv;
    std::vector<int64_t> wtb, wbnd;
    for (size_t a : ord) {
        const PairGeo &G = geo[a];
        const int64_t pb = band_bnd_bytes(G.bnd);
        int best = -1;
        for (size_t k = 0; k < wv.size(); ++k) {
            if (wtb[k] + G.tb <= cap_tb && wbnd[k] + pb <= cap_bnd &&
                (best < 0 || wbnd[k] * cap_tb + wtb[k] * cap_bnd < wbnd[best] * cap_tb + wtb[best] * cap_bnd))
                best = (int)k;
        }
        if (best < 0) {
            wv.emplace_back();
            wtb.push_back(0), wbnd.push_back(0);
            best = (int)wv.size() - 1;
        }
        wtb[best] += G.tb, wbnd[best] += pb;
        wv[best].push_back(a);
    }
    struct U {
        int64_t start;
        int slot, s;
    };
    auto by_start = [](const U &x, const U &y) {
        return x.start != y.start ? x.start < y.start : (x.slot != y.slot ? x.slot < y.slot : x.s < y.s);
    };
    for (size_t k = 0; k < wv.size(); ++k) {
        BandWave W;
        W.pair0 = (int)bp.pairs.size(), W.npair = (int)wv[k].size();
        W.unit0 = (int)bp.units.size(), W.strip0 = (int)bp.strips.size();
        int64_t tb = 0, bnd = 0;
        std::vector<U> us;
        std::vector<std::pair<int, size_t>> ck;  // (slot, geo index) of the recomputed pairs
        for (size_t a : wv[k]) {
            const PairGeo &G = geo[a];
            const KswPair &kp = pairs[G.id];
            BandPairDev pd;
            pd.qoff = kp.qoff, pd.toff = kp.toff, pd.cig_off = kp.cig_off;
            pd.qlen = kp.qlen, pd.tlen = kp.tlen, pd.w = G.ww, pd.rb = G.rb;
            pd.strip0 = (int)bp.strips.size();
            pd.nstrip = (int)G.strips.size();
            pd.idx = G.id, pd.ckpt = G.ckpt ? 1 : 0;
            const int slot = (int)bp.pairs.size();
            bp.pairs.push_back(pd);
            for (size_t s = 0; s < G.strips.size(); ++s) {
                BandStripDev sd = G.strips[s];
                if (!G.ckpt) sd.tb_off += tb;
                sd.bnd_off += bnd;
                bp.strips.push_back(sd);
                us.push_back(U{G.start[s], slot, (int)s});
            }
            if (G.ckpt && !G.notb) ck.push_back({slot, a});
            tb += G.tb;
            bnd += (G.bnd + 31) / 32 * 32;
        }
        // strips in estimated start order; a pair's strips keep their left-to-right order
        std::stable_sort(us.begin(), us.end(), by_start);
        for (const U &x : us) bp.units.push_back(make_int2(x.slot, x.s));
        W.nunit = (int)us.size();
        W.nstrip = (int)bp.strips.size() - W.strip0;
        W.tb_bytes = tb, W.bnd_entries = bnd;
        bp.tb_cap = std::max(bp.tb_cap, tb);
        bp.bnd_cap = std::max(bp.bnd_cap, bnd);
        // Recompute rounds: each recomputed pair gets a share of the round budget in proportion
        // to its whole traceback (so that all pairs need about as many rounds) and is cut into
        // groups of consecutive strips within it (at least one strip); round r recomputes the
        // r-th group from the right of every pair that has one, all together.
        W.round0 = (int)bp.rounds.size();
        std::vector<std::vector<std::pair<int, int>>> groups(ck.size());  // per pair: [s0, s1) right to left
        std::vector<std::vector<int64_t>> gtb(ck.size());
        double tb_all = 0;
        for (size_t c = 0; c < ck.size(); ++c)
            for (int64_t x : geo[ck[c].second].stb) tb_all += (double)x;
        size_t nround = 0;
        for (size_t c = 0; c < ck.size(); ++c) {
            const PairGeo &G = geo[ck[c].second];
            double tb_pair = 0;
            for (int64_t x : G.stb) tb_pair += (double)x;
            const int64_t share = std::max<int64_t>((int64_t)((double)gres * tb_pair / std::max(tb_all, 1.0)), 1);
            int s1 = (int)G.strips.size();
            while (s1 > 0) {
                int s0 = s1 - 1;
                int64_t acc = G.stb[s0];
                while (s0 > 0 && acc + G.stb[s0 - 1] <= share) acc += G.stb[--s0];
                groups[c].push_back({s0, s1});
                gtb[c].push_back(acc);
                s1 = s0;
            }
            nround = std::max(nround, groups[c].size());
        }
        for (size_t r = 0; r < nround; ++r) {
            BandRound R;
            R.group0 = (int)bp.groups.size(), R.unit0 = (int)bp.units.size(), R.nstrip = 0;
            int64_t off = 0;
            std::vector<U> ru;
            for (size_t c = 0; c < ck.size(); ++c) {
                if (r >= groups[c].size()) continue;
                const int slot = ck[c].first;
                const PairGeo &G = geo[ck[c].second];
                const BandPairDev &pd = bp.pairs[slot];
                const int s0 = groups[c][r].first, s1 = groups[c][r].second;
                BandGroupDev gd;
                gd.slot = slot, gd.s_first = pd.strip0 + s0, gd.s_end = pd.strip0 + s1;
                gd.col_lo = s0 * SW;
                gd.last = r + 1 == groups[c].size() ? 1 : 0;
                gd.pad = 0;
                bp.groups.push_back(gd);
                int64_t o = off;
                for (int s = s0; s < s1; ++s) {
                    bp.strips[pd.strip0 + s].tb_off = o;  // this round's arena
                    o += G.stb[s];
                    ru.push_back(U{G.start[s] - G.start[s0], slot, s});
                }
                off += gtb[c][r];
                R.nstrip += s1 - s0;
            }
            std::stable_sort(ru.begin(), ru.end(), by_start);
            for (const U &x : ru) bp.units.push_back(make_int2(x.slot, x.s));
            R.ngroup = (int)bp.groups.size() - R.group0;
            R.nunit = (int)ru.size();
            R.tb_bytes = off;
            bp.tb_cap = std::max(bp.tb_cap, off);
            bp.rounds.push_back(R);
        }
        W.nround = (int)bp.rounds.size() - W.round0;
        bp.waves.push_back(W);
    }
    return 0;
}

int band_occupancy(int flag) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, band_kernel_for(flag, 64), 256, 0) != cudaSuccess) return 1;
    return std::max(nb, 1);
}

cudaError_t band_launch_units(const BandPlan &bp, const BandArgs &a, int flag, int ctas, cudaStream_t st);

cudaError_t band_launch_dp(const BandPlan &bp, int k, const BandDev &D, const uint8_t *qcodes,
                           const uint8_t *tcodes, const KswScore &S, int flag, int ctas, cudaStream_t st) {
    const BandWave &W = bp.waves[k];
    cudaError_t e;
    // no boundary entry is written yet
    if ((e = cudaMemsetAsync(D.bnd, 0, sizeof(uint2) * (size_t)W.bnd_entries, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(D.res + W.pair0, 0, sizeof(BandRes) * std::max(W.npair, 1), st)) != cudaSuccess)
        return e;
    if ((e = cudaMemsetAsync(D.queue + 64 * k, 0, sizeof(int32_t), st)) != cudaSuccess) return e;
    BandArgs a;
    a.qcodes = qcodes, a.tcodes = tcodes;
    a.pairs = D.pairs, a.strips = D.strips, a.units = D.units + W.unit0;
    a.n_units = W.nunit;
    a.queue = D.queue + 64 * k, a.error = D.error;
    a.tb = D.tb, a.bnd = D.bnd, a.res = D.res;
    a.sc = S;
    a.block = bp.block;
    a.generic = (flag & AW_EZ_GENERIC_SC) ? 1 : 0;
    a.sse_st = (flag & AW_EZ_SINGLETRACK) && (flag & AW_EZ_SSE_SINGLETRACK) ? 1 : 0;
    a.store_ckpt = 0;
    a.deadline = D.deadline;
    a.walk = nullptr;
    return band_launch_units(bp, a, flag, ctas, st);
}

cudaError_t band_launch_units(const BandPlan &bp, const BandArgs &a, int flag, int ctas, cudaStream_t st) {
    const bool cigar = !(flag & AW_EZ_SCORE_ONLY), right = !!(flag & AW_EZ_RIGHT);
    const bool stk = cigar && singletrack_tracks(flag, bp.block);
    const int grid = std::max(1, std::min(ctas, (a.n_units + 7) / 8));
#define AW_BAND_LAUNCH(NCV)                                                                   \
    if (stk) ksw_band_kernel<true, false, true, NCV><<<grid, 256, 0, st>>>(a);               \
    else if (cigar && right) ksw_band_kernel<true, true, false, NCV><<<grid, 256, 0, st>>>(a); \
    else if (cigar) ksw_band_kernel<true, false, false, NCV><<<grid, 256, 0, st>>>(a);        \
    else ksw_band_kernel<false, false, false, NCV><<<grid, 256, 0, st>>>(a);
    if (bp.nc == 4) {
        AW_BAND_LAUNCH(4)
    } else {
        AW_BAND_LAUNCH(8)
    }
#undef AW_BAND_LAUNCH
    return cudaGetLastError();
}

cudaError_t band_launch_finish(const BandPlan &bp, int k, const BandDev &D, const uint8_t *qcodes,
                               const uint8_t *tcodes, const KswScore &S, int flag, KswOut *out, uint32_t *cig,
                               const int8_t *mat, int m, cudaStream_t st) {
    const BandWave &W = bp.waves[k];
    BtArgs b;
    b.pairs = D.pairs + W.pair0, b.npair = W.npair, b.strips = D.strips, b.tb = D.tb, b.res = D.res + W.pair0;
    b.walk = D.walk + W.pair0;
    b.qcodes = qcodes, b.tcodes = tcodes, b.out = out, b.cig = cig, b.sc = S;
    memset(b.mat, 0, sizeof(b.mat));
    memcpy(b.mat, mat, (size_t)m * m);
    b.m = m, b.flag = flag, b.block = bp.block;
    const bool stk = singletrack_tracks(flag, b.block) && !(flag & AW_EZ_SCORE_ONLY);
    const int fw = stk ? fin_warps<true>() : fin_warps<false>();
    const int grid = (W.npair + fw - 1) / fw;
    if (bp.nc == 4) {
        if (stk) ksw_band_finish_kernel<true, 4><<<grid, 32 * fw, 0, st>>>(b);
        else ksw_band_finish_kernel<false, 4><<<grid, 32 * fw, 0, st>>>(b);
    } else {
        if (stk) ksw_band_finish_kernel<true, 8><<<grid, 32 * fw, 0, st>>>(b);
        else ksw_band_finish_kernel<false, 8><<<grid, 32 * fw, 0, st>>>(b);
    }
    return cudaGetLastError();
}

cudaError_t band_launch_groups(const BandPlan &bp, int k, const BandDev &D, const uint8_t *qcodes,
                               const uint8_t *tcodes, const KswScore &S, int flag, KswOut *out, uint32_t *cig,
                               const int8_t *mat, int m, int ctas, cudaStream_t st) {
    const BandWave &W = bp.waves[k];
    cudaError_t e;
    BtArgs b;
    b.pairs = D.pairs, b.npair = (int)bp.pairs.size(), b.strips = D.strips, b.tb = D.tb, b.res = D.res;
    b.walk = D.walk;
    b.qcodes = qcodes, b.tcodes = tcodes, b.out = out, b.cig = cig, b.sc = S;
    memset(b.mat, 0, sizeof(b.mat));
    memcpy(b.mat, mat, (size_t)m * m);
    b.m = m, b.flag = flag, b.block = bp.block;
    for (int ri = W.round0; ri < W.round0 + W.nround; ++ri) {
        const BandRound &R = bp.rounds[ri];
        const BandGroupDev *gd = D.groups + R.group0;
        // every strip's left column is there from the first pass, so the strips of a round do
        // not wait for one another
        // this round's counter of the work queue: the wave's slot, reused per round
        if ((e = cudaMemsetAsync(D.queue + 64 * k, 0, sizeof(int32_t), st)) != cudaSuccess) return e;
        BandArgs a;
        a.qcodes = qcodes, a.tcodes = tcodes;
        a.pairs = D.pairs, a.strips = D.strips, a.units = D.units + R.unit0;
        a.n_units = R.nunit;
        a.queue = D.queue + 64 * k, a.error = D.error;
        a.tb = D.tb, a.bnd = D.bnd, a.res = D.res;
        a.sc = S;
        a.block = bp.block;
        a.generic = (flag & AW_EZ_GENERIC_SC) ? 1 : 0;
        a.sse_st = (flag & AW_EZ_SINGLETRACK) && (flag & AW_EZ_SSE_SINGLETRACK) ? 1 : 0;
        a.store_ckpt = 1;
        a.deadline = D.deadline;
        a.walk = D.walk;
        if ((e = band_launch_units(bp, a, flag, ctas, st)) != cudaSuccess) return e;
        if (bp.nc == 4) ksw_band_round_walk_kernel<4><<<R.ngroup, 32, 0, st>>>(b, gd);
        else ksw_band_round_walk_kernel<8><<<R.ngroup, 32, 0, st>>>(b, gd);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace aw
