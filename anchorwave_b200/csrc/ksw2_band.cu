// KSW2 extd2, banded form (w >= 0) and the Singletrack traceback, on sm_100a.
//
// The reference sweeps anti-diagonals r and keeps the int8 difference cells in
// arrays indexed by target position t; on each anti-diagonal it recomputes whole
// SIMD blocks [stB, en16] (st0 rounded down to the block, en0 rounded up to 16),
// so cells just outside the band ("padding") are computed from whatever the arrays
// held, and the in-band cells and the traceback read them
// (minimap2/ksw2_extd2_avx.c:255-701, ksw2_extd2_sse.c:136-331).  This kernel
// computes the same cells in target-column strips, one warp per strip, which sweeps the
// anti-diagonals as the reference does: at step r lane L holds the cells of its columns on
// anti-diagonal r, two per register (ksw2_cell.cuh), and the registers of a column are the
// reference's arrays at its position:
//   * the cells of a step do not depend on one another, so a step costs one cell's latency
//     and a warp alone keeps its scheduler busy (a sweep by rows, each lane's cells a serial
//     chain, took 0.61 us per 4-column step at the band's edge, one anti-diagonal takes 0.25);
//   * st0, en0 and the blocks around them are the same for the whole warp, and a lane's columns
//     lie in one 16-column block, so "computed" is a property of a lane: a lane outside
//     [st16, en16] skips its cells and its registers keep their last values;
//   * left input of cell (t, r): the column t-1 at r-1 (the previous lane's last column by a
//     shuffle); at t == st16 the reference's boundary value (x[st16-1] only on the anti-diagonal
//     where st16 advanced, constants otherwise, the matrix edge when st16 == 0,
//     ksw2_extd2_avx.c:273-287);
//   * up input: the column's own registers, the top-edge values on row 0;
//   * score: the score-fill (ksw2_extd2_avx.c:289-311) refreshes position t on
//     anti-diagonal r when st0 <= t <= st0+16*ceil((en0-st0+1)/16)-1 (en0 for
//     generic scoring); otherwise the stale value of the last fill stays.  Query codes move
//     one column per step with the cells (code 0 above the matrix);
//   * H row: H[t] += v[t] inside the band, H[en0] = H[en0-1] + u[en0] on the right
//     edge (ksw2_extd2_sse.c:332-367), mqe/mte with ">=" (:369-372), the score
//     on the last anti-diagonal; the anti-diagonal loop stops at the first empty
//     band (:151-154, zdropped = 1).
// Cells above the matrix, below it and right of it that a lane computes along with its others
// never reach a cell of the matrix.
//
// The blocks left of st16 that the reference computes as well (blocks of 32 or 64 bytes) feed no
// cell from st16 on, and only a traceback that leaves the band by more than its last 16-column
// block reads them (89 of 420,000 walks in bands of 1 to 24 around random, shifted and gapped
// pairs), while their y and y2 grow without a bound of use (by q + e - e2 a step: 629 under (4, 2,
// 24, 1), 4,150 under (30, 4, 40, 1), beyond a 16-bit field).  So the sweep leaves them out: when
// st16 passes a block its columns' state is stored (DeepRows), and a walk that gets there
// computes the cells from it in 32 bits (deep_fill).
//
// Three ranges of a strip's steps, solved once per strip, run on
// loops of their own: the steps where the whole strip lies strictly inside the band (no
// tests), before them those where only the band's right edge is in the strip, and after them
// those with only its left edge.  Both edges are chains that bound long pairs: every step of
// a pair has some strip at each of them.  H is kept where a later step needs it: not at all
// while the right edge is in the strip (it follows from the left column's H and the u and v
// of an anti-diagonal), for the lane's last column afterwards (the others follow in the same
// way).
//
// Work decomposition: every (pair, strip) is a unit of a device queue, ordered so
// that a strip is always taken after the strip on its left, and reads its left column as that
// strip writes it.  The band enters a strip SW columns further right 2 SW steps later, so a
// long pair takes about two steps per target base whatever the strip's width, and its strips
// run on as many warps, across CTAs, as the band is high.  An entry of a boundary column
// carries a mark that says it is written (the columns are cleared before the first pass), so
// a strip reads eight rows ahead and waits (bounded) only for entries that are not there yet:
// no fence and no counter between the strips.
#include "ksw2_band.h"
#include "ksw2_cell.cuh"
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

__device__ __forceinline__ int prmt_sx(uint32_t lo, uint32_t hi, uint32_t sel) { return (int)prmt(lo, hi, sel); }
__device__ __forceinline__ int sx8(uint32_t w) { return (int)(int8_t)(uint8_t)w; }
__device__ __forceinline__ uint32_t pack3(int a, int b, int c) {
    return (uint32_t)(a & 0xff) | ((uint32_t)(b & 0xff) << 8) | ((uint32_t)(c & 0xff) << 16);
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
    uint32_t one = 1;  // KswFullArgs::one
    int peak_max;      // largest field of x, y, x2, y2 (as often as they are checked) that keeps the cells exact
};

constexpr uint64_t WAIT_NS = 20ull * 1000 * 1000 * 1000;  // bounded wait on the left strip
// Rows of the left column read at a time.
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

// Value of a field of 16 * value + FB (+ tag).
__device__ __forceinline__ int fval(uint32_t w, int f) { return (fld(w, f) - FB) >> 4; }
// Both fields of a pair from two conditions.
__device__ __forceinline__ uint32_t mask2(bool lo, bool hi) { return (lo ? 0xffffu : 0u) | (hi ? 0xffff0000u : 0u); }

// The traceback words of a step.  A word holds four columns of one row, whose cells lie on four
// consecutive anti-diagonals: the bytes of the first three columns wait for the fourth.  put()
// takes a byte per field (bits 0-7 and 16-23 of d[p]: columns p and p + NP) and returns the
// word completed at this step, of row r - 3 - (its first column).
struct RowWords {  // columns 0, 2 in d[0]; 1, 3 in d[1]
    uint32_t a0 = 0, a1 = 0, a2 = 0;
    __device__ __forceinline__ uint32_t put(const uint32_t (&d)[2]) {
        const uint32_t w = prmt(a2, d[1], 0x6210);
        a2 = prmt(a1, d[0], 0x7610);
        a1 = prmt(a0, d[1], 0x5540);
        a0 = d[0];
        return w;
    }
};

// A lane holds C = 4 target columns in NP pairs; a strip is SW = 128 columns.  (Eight columns per
// lane took 0.45 us a step against 0.25 and were no faster on 512 pairs of 5 kb at w = 50%,
// which are bound by their work: 15.4 against 14.1 ms.)
constexpr int NP = 2, C = 2 * NP, SW = 32 * C;
// Traceback layout: words of 4 columns (state bytes, or v then u bytes), NG words per slot.  The
// word of group g (columns 4g..4g+3 of the strip) and row j lies in slot (j - jlo) + 4g from the
// strip's start.  The next strip of the pair starts after as many slots as this one has rows: the
// corner that the skew leaves free at its start is where this one's last rows end.
constexpr int NG = SW / 4;

// The state of the columns that st16 passes (this comment's "deep" cells: columns below st16 of its
// block), stored as further rows of the strip's traceback: 14 words of a lane's registers, then
// a word that is 1 once the block's bytes are computed (in the block's first lane).
template <int WB>
struct DeepRows {
    static constexpr int WORDS = 14;
    // word w of lane l of a strip
    static __device__ __forceinline__ uint32_t *word(uint8_t *tb, const BandStripDev &St, int l, int w) {
        const int row = St.jend - St.jlo + 1 + w * 4 / WB;
        return reinterpret_cast<uint32_t *>(tb + St.tb_off + ((int64_t)(row + 4 * l) * NG + l) * WB + w * 4 % WB);
    }
};
// Whether a pair's walk can meet one: not in 16-byte blocks, nor in bands that no column leaves.
__host__ __device__ inline bool deep_cells(int block, int w, int qlen) { return block > 16 && w < qlen; }

constexpr int BAND_WARPS = 4;  // per CTA: small CTAs spread a pair's strips over the SMs
// CTAs per SM that the registers are sized for.  With the state bytes the edge loops want more than
// the 128 registers of four CTAs (one 160 kb pair at w = 10% 104 against 95 ms of sweep with three, 512
// pairs of 5 kb at 250 5.0 / 4.6), which batches of many narrow bands pay for (2,000 of 2 kb at 50: 3.8 /
// 4.1); the tracks and the score alone do not.
constexpr int band_ctas(int mode) { return mode == LEFT || mode == RIGHTMOST ? 3 : 4; }

// STRICT: every step's values are checked, not those of every PUB-th step (band_strict).
template <int MODE, bool STRICT>
__global__ void __launch_bounds__(32 * BAND_WARPS, band_ctas(MODE)) ksw_band_kernel(BandArgs A) {
    constexpr bool CIGAR = MODE != SCORES;
    constexpr int WB = MODE == TRACKS ? 8 : 4;
    using T = Tags<MODE>;
    const int lane = threadIdx.x & 31;
    const KswScore &S = A.sc;
    const CellK K = make_cellk<MODE>(S, A.one);
    const int B = A.block;

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
        const int c0 = s * SW, col0 = c0 + lane * C, rs = c0 + jstart;
        const bool last_strip = s + 1 == P.nstrip;
        // the strip on the left and its stored rows; on other rows (and for an empty strip) the
        // arrays' initial values, which no cell of the band reads
        int prod_lo = 0, prod_hi = -1;
        const uint2 *bnd_prod = nullptr;
        if (s > 0) {
            const BandStripDev Pr = A.strips[P.strip0 + s - 1];
            prod_lo = Pr.jlo, prod_hi = min(Pr.jend, wlim);
            bnd_prod = A.bnd + Pr.bnd_off;
        }
        // a recompute round reads the columns of the first pass and writes none
        uint2 *bnd_me = lane == 31 && !last_strip && !A.walk ? A.bnd + St.bnd_off : nullptr;
        const bool store_tb = CIGAR && (!P.ckpt || A.store_ckpt);  // this strip's traceback is kept
        // this lane's word completed at step 0 (row rs - c0 - 3 of group 0, slot jstart - 3 - jlo), and
        // its stored row; only words of stored rows are written, the slots are shared with others
        const int slot0 = jstart - 3 - jlo, row0 = slot0 - 4 * lane;
        const unsigned nrows = col0 < tlen ? (unsigned)(St.jend - jlo + 1) : 0u;
        uint8_t *tbp = CIGAR ? A.tb + St.tb_off + ((int64_t)slot0 * NG + lane) * WB : nullptr;
        const bool deep = CIGAR && store_tb && deep_cells(B, w, qlen);
        BandRes *R = A.res + un.x;
        // steps whose cells all lie strictly inside the band
        const int ri0 = max(c0 + SW, 2 * (c0 + SW) - w);
        const int ri1 = min(min(rlim - 1, c0 + qm1 - 1), c0 > 0 ? 2 * c0 + w - 2 : w);
        const int kf0 = ri0 - rs, kf1 = c0 + SW <= tm1 ? ri1 - rs + 1 : 0;
        // in the last strip, from the step after the last column entered the band
        const int kz0 = max(tm1, 2 * tm1 - w) + 1 - rs, kz1 = last_strip ? ri1 - rs + 1 : 0;
        // the steps after kf0 whose left edge may lie in the strip
        const int kl1 = c0 + SW <= tm1 ? min(rlim, c0 + qm1) - rs : 0;
        // steps below row 0 with the left edge (st0) left of the strip and the right edge before its
        // last column, whose H the strip on the right reads from then on
        const int kr0 = c0 + SW - rs, kr1 = c0 > 0 ? min(kf1, 2 * (c0 + SW - 1) - w - rs) : 0;
        // the last step: the strip's last word of row jend
        const int nsteps = c0 + min(SW, ((tlen - c0) + 3) & ~3) - 1 + jend - rs + 1;

        uint32_t X[NP], V[NP], X2[NP], U[NP], Y[NP], Y2[NP], SS[NP];
        uint32_t rlo[C], rhi[C], sel[C];
        int H[C];
        const uint32_t x_in = K.kxa, v_in = rep2(FB - 16 * S.qe), x2_in = K.kxa2;  // initial values
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int t = col0 + c;
            const int tc = t < tlen ? (ts[t] & 7) : 0;
            rlo[c] = S.tab_lo[tc];
            rhi[c] = S.tab_hi[tc];
            sel[c] = 0x8880u;  // query code 0
            H[c] = AW_NEG_INF;
        }
        constexpr int SB = T::s + 2 * FB;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            X[p] = x_in, V[p] = v_in, X2[p] = x2_in;
            U[p] = v_in, Y[p] = K.kxb, Y2[p] = K.kxb2;
            SS[p] = add2(SB);  // score 0
        }
        uint32_t peak = 0;  // the largest x, y, x2, y2 field so far
        RowWords words, words2;
        enum { H_NONE, H_LAST, H_ALL };
        int h_state = H_ALL;             // the columns whose H is up to date
        unsigned long long mte_key = 0;  // last strip: the lane that owns the last column
        const int pm = A.sse_st ? INT_MAX : 0;  // strict end rule: mirrored positions
        // lane 0's left values of row jr: x, v, x2 with the mark, and the H on the left
        auto left_of = [&](int jr) -> uint2 {
            if (s == 0) return make_uint2(pack3(-S.qe, edge_diff(jr, S), -S.qe2) | BND_MARK, (uint32_t)AW_NEG_INF);
            if (jr < prod_lo || jr > prod_hi) return make_uint2(pack3(-S.qe, -S.qe, -S.qe2) | BND_MARK, (uint32_t)AW_NEG_INF);
            return bnd_load(bnd_prod + (jr - prod_lo));
        };
        // the score selector of row jr's query code
        auto code_of = [&](int jr) -> uint32_t { return (jr >= 0 && jr < qlen ? qs[jr] & 7u : 0u) * 0x1111u + 0x8880u; };
        // lane i holds what lane 0 needs for row jstart + (k & ~31) + i: the next group's entries
        // and the next 32 query codes are on their way while the current ones are used
        uint2 ahead = make_uint2(BND_MARK, 0u);
        if (lane < PUB) ahead = left_of(jstart + lane);
        uint32_t qnext = code_of(jstart + lane), qcur = 0, bx = 0, by = 0;
        int bh = 0;
        bool failed = false, stopped = false;
        // the words of step k into the traceback
        auto store_words = [&](const uint32_t (&d)[NP], const uint32_t (&d2)[NP], uint8_t *dst, int k) {
            const uint32_t a = words.put(d);
            if constexpr (MODE == TRACKS) {
                const uint32_t b = words2.put(d2);
                if ((unsigned)(row0 + k) < nrows) __stcs(reinterpret_cast<uint2 *>(dst), make_uint2(a, b));
            } else {
                if ((unsigned)(row0 + k) < nrows) __stcs(reinterpret_cast<uint32_t *>(dst), a);
            }
        };
        // no candidate before the next call can leave its field while these stay below peak_max
        auto grown = [&]() {
#pragma unroll
            for (int p = 0; p < NP; ++p)
                peak = __vimax3_s16x2(peak, X[p], X2[p]), peak = __vimax3_s16x2(peak, Y[p], Y2[p]);
        };
        // the columns of the 16 that st16 has just passed, before the first step without them
        auto store_deep = [&](int st16) {
            if ((st16 & (B - 1)) == 0 || (col0 & ~15) != st16 - 16) return;
            // DeepRows::word by what the warp has in registers
            uint8_t *at = tbp + (int64_t)((int)nrows - row0) * (NG * WB);
            const uint32_t st[DeepRows<WB>::WORDS + 1] = {X[0],  X[1], V[0],  V[1],  X2[0], X2[1], U[0], U[1],
                                                          Y[0],  Y[1], Y2[0], Y2[1], SS[0], SS[1], 0u};
#pragma unroll
            for (int i = 0; i <= DeepRows<WB>::WORDS; ++i)
                *reinterpret_cast<uint32_t *>(at + i * 4 / WB * (NG * WB) + i * 4 % WB) = st[i];
        };
        // the last column's entry: x, v, x2 as bytes (a field's bits 4-11) and H
        auto store_entry = [&](uint2 *dst) {
            const uint32_t a = prmt(X[NP - 1], V[NP - 1], 0x7632) >> 4, b = X2[NP - 1] >> 4;
            bnd_store(dst, prmt(a, b, 0x6620) & 0xffffffu, (uint32_t)H[C - 1]);
        };
        auto score_of = [&](int p) -> uint32_t {
            return (uint32_t)prmt_sx(rlo[p + NP], rhi[p + NP], sel[p + NP]) * (16u << 16) +
                   ((uint32_t)prmt_sx(rlo[p], rhi[p], sel[p]) * 16u + add2(SB));
        };
        // H of every column in the band after step k-1, from the left column's H at that step:
        // H(t, j) = H(t-1, j) + u(t, j), and along the anti-diagonal H(t+1, j-1) = H(t, j) - v(t, j)
        // + u(t+1, j-1)
        auto rebuild_h = [&](int k) {
            int sum = 0;
#pragma unroll
            for (int c = 0; c < C; ++c) sum += fval(U[c % NP], c / NP) - fval(V[c % NP], c / NP);
            int before = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, before, o);
                if (lane >= o) before += t;
            }
            int h = __shfl_sync(FULL, bh, (k - 1) & 31) + before - sum;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                h += fval(U[c % NP], c / NP);
                H[c] = h;
                h -= fval(V[c % NP], c / NP);
            }
        };
        // The lane's other columns from the last one's: along the anti-diagonal,
        // H(t, j) = H(t+1, j-1) - u(t+1, j-1) + v(t, j)
        auto h_from_last = [&]() {
#pragma unroll
            for (int c = C - 2; c >= 0; --c)
                H[c] = H[c + 1] - fval(U[(c + 1) % NP], (c + 1) / NP) + fval(V[c % NP], c / NP);
        };
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
            if (mine) {
                bx = (uint32_t)(16 * sx8(ahead.x) + FB + T::a) | (uint32_t)(16 * sx8(ahead.x >> 8) + FB) << 16;
                by = (uint32_t)(16 * sx8(ahead.x >> 16) + FB + T::a2) | qcur << 16;
                bh = (int)ahead.y;
            }
            if ((lane & ~(PUB - 1)) == ((kb + PUB) & 31)) ahead = left_of(jstart + ((kb + PUB) & ~31) + lane);
            if (!STRICT) grown();
            const int kend = min(kb + PUB, nsteps);
            const bool full = kend - kb == PUB;  // the loops below take whole groups, unrolled
            int k = kb;
            uint8_t *tb = tbp + (int64_t)kb * (NG * WB);
            // the last column's entry of the group's first row, and the rows it may be stored for
            const int je0 = rs + kb - (c0 + SW - 1);
            uint2 *entry = bnd_me + (je0 - jlo);
            const bool entries = !last_strip && !A.walk && je0 + PUB > jlo && je0 <= jend;
            if (full && ((k >= kf0 && kend <= kf1) || (k >= kz0 && kend <= kz1))) {
                // interior: no tests inside the group
                if (h_state == H_NONE) rebuild_h(k);
                if (last_strip && h_state == H_LAST) h_from_last();
                h_state = last_strip ? H_ALL : H_LAST;
#pragma unroll 4
                for (int i = 0; i < PUB; ++i) {
                    uint32_t r0 = __shfl_up_sync(FULL, prmt(X[NP - 1], V[NP - 1], 0x7632), 1);
                    uint32_t r1 = __shfl_up_sync(FULL, prmt(X2[NP - 1], sel[C - 1], 0x5432), 1);
                    const uint32_t b0 = __shfl_sync(FULL, bx, (kb & 31) + i), b1 = __shfl_sync(FULL, by, (kb & 31) + i);
                    if (lane == 0) r0 = b0, r1 = b1;
                    uint32_t x = prmt(r0, X[NP - 1], 0x5410), v = prmt(r0, V[NP - 1], 0x5432), x2 = prmt(r1, X2[NP - 1], 0x5410);
#pragma unroll
                    for (int c = C - 1; c > 0; --c) sel[c] = sel[c - 1];
                    sel[0] = r1 >> 16;
                    uint32_t d[NP], d2[NP];
#pragma unroll
                    for (int p = NP - 1; p >= 0; --p) {
                        uint32_t xp = p ? X[p - 1] : x, vp = p ? V[p - 1] : v, x2p = p ? X2[p - 1] : x2;
                        SS[p] = score_of(p);
                        cell2<MODE, true>(SS[p], xp, vp, x2p, U[p], Y[p], Y2[p], d[p], K);
                        X[p] = xp, V[p] = vp, X2[p] = x2p;
                        if (MODE == TRACKS) d[p] = vp >> 4, d2[p] = U[p] >> 4;
                    }
                    if (last_strip) {
                        // H of the last column (all columns are kept here, for the last row)
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            H[c] += fval(V[c % NP], c / NP);
                            if (col0 + c == tm1) {
                                const unsigned long long key = end_key(H[c], pm ^ (rs + kb + i - tm1));
                                mte_key = key > mte_key ? key : mte_key;
                            }
                        }
                    } else {
                        H[C - 1] += fval(V[NP - 1], 1);
                    }
                    if (STRICT) grown();
                    if (CIGAR && store_tb) store_words(d, d2, tb + i * (NG * WB), kb + i);
                    if (entries && bnd_me) store_entry(entry + i);
                }
                continue;
            }
            if (full && k >= kf0 && kend <= kl1) {
                // the left edge alone: which lanes are computed, the first one's left input, and
                // where the fill starts
                if (h_state == H_NONE) rebuild_h(k);
                h_state = H_LAST;
                // the group in two parts when st16 advances in it (with a test and the stores in
                // each step one 100 kb pair at w = 10 kb took 69.7 ms of sweep, like this 61.7)
                const int adv = -(rs + kb - w + 1) & 31;
                int i = 0;
                for (int to = deep && adv < PUB ? adv : PUB;; to = PUB) {
#pragma unroll 2
                    for (; i < to; ++i) {
                        const int r = rs + kb + i, st0 = max((r - w + 1) >> 1, 0), st16 = st0 & ~15;
                        uint32_t r0 = __shfl_up_sync(FULL, prmt(X[NP - 1], V[NP - 1], 0x7632), 1);
                        uint32_t r1 = __shfl_up_sync(FULL, prmt(X2[NP - 1], sel[C - 1], 0x5432), 1);
                        const uint32_t b0 = __shfl_sync(FULL, bx, (kb & 31) + i), b1 = __shfl_sync(FULL, by, (kb & 31) + i);
                        if (lane == 0) r0 = b0, r1 = b1;
#pragma unroll
                        for (int c = C - 1; c > 0; --c) sel[c] = sel[c - 1];
                        sel[0] = r1 >> 16;
                        const bool fix = col0 == st16 && st16 > 0 && ((max((r - w) >> 1, 0)) & ~15) == st16;
                        if (fix) r0 = prmt(x_in, v_in, 0x5410), r1 = x2_in;
                        const uint32_t x = prmt(r0, X[NP - 1], 0x5410), v = prmt(r0, V[NP - 1], 0x5432), x2 = prmt(r1, X2[NP - 1], 0x5410);
                        uint32_t d[NP], d2[NP];
                        const int f0 = st0 - col0;
#pragma unroll
                        for (int p = 0; p < NP; ++p) {
                            const uint32_t m = mask2(p >= f0, p + NP >= f0);
                            SS[p] = (score_of(p) & m) | (SS[p] & ~m);
                            d[p] = d2[p] = 0;
                        }
                        if (col0 >= st16) {
#pragma unroll
                            for (int p = NP - 1; p >= 0; --p) {
                                uint32_t xp = p ? X[p - 1] : x, vp = p ? V[p - 1] : v, x2p = p ? X2[p - 1] : x2;
                                cell2<MODE, true>(SS[p], xp, vp, x2p, U[p], Y[p], Y2[p], d[p], K);
                                X[p] = xp, V[p] = vp, X2[p] = x2p;
                                if (MODE == TRACKS) d[p] = vp >> 4, d2[p] = U[p] >> 4;
                            }
                            if (f0 < C) H[C - 1] += fval(V[NP - 1], 1);
                        }
                        if (STRICT) grown();
                        if (CIGAR && store_tb) store_words(d, d2, tb + i * (NG * WB), kb + i);
                        if (entries && bnd_me && je0 + i <= jend) store_entry(entry + i);
                    }
                    if (to == PUB) break;
                    store_deep(max((rs + kb + i - w + 1) >> 1, 0) & ~15);
                }
                continue;
            }
            if (full && k >= kr0 && kend <= kr1) {
                // the right edge alone: which lanes are computed, and how far the fill reaches
                h_state = H_NONE;
#pragma unroll 2
                for (int i = 0; i < PUB; ++i) {
                    const int r = rs + kb + i, en0 = (r + w) >> 1, st0 = max(r - qm1, (r - w + 1) >> 1);
                    const int f1 = (A.generic ? en0 : st0 + ((en0 - st0 + 16) & ~15) - 1) - col0;
                    uint32_t r0 = __shfl_up_sync(FULL, prmt(X[NP - 1], V[NP - 1], 0x7632), 1);
                    uint32_t r1 = __shfl_up_sync(FULL, prmt(X2[NP - 1], sel[C - 1], 0x5432), 1);
                    const uint32_t b0 = __shfl_sync(FULL, bx, (kb & 31) + i), b1 = __shfl_sync(FULL, by, (kb & 31) + i);
                    if (lane == 0) r0 = b0, r1 = b1;
                    const uint32_t x = prmt(r0, X[NP - 1], 0x5410), v = prmt(r0, V[NP - 1], 0x5432), x2 = prmt(r1, X2[NP - 1], 0x5410);
#pragma unroll
                    for (int c = C - 1; c > 0; --c) sel[c] = sel[c - 1];
                    sel[0] = r1 >> 16;
                    uint32_t d[NP], d2[NP];
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        const uint32_t m = mask2(p <= f1, p + NP <= f1);
                        SS[p] = (score_of(p) & m) | (SS[p] & ~m);
                        d[p] = d2[p] = 0;
                    }
                    if (col0 <= (en0 | 15)) {
#pragma unroll
                        for (int p = NP - 1; p >= 0; --p) {
                            uint32_t xp = p ? X[p - 1] : x, vp = p ? V[p - 1] : v, x2p = p ? X2[p - 1] : x2;
                            cell2<MODE, true>(SS[p], xp, vp, x2p, U[p], Y[p], Y2[p], d[p], K);
                            X[p] = xp, V[p] = vp, X2[p] = x2p;
                            if (MODE == TRACKS) d[p] = vp >> 4, d2[p] = U[p] >> 4;
                        }
                    }
                    if (STRICT) grown();
                    if (CIGAR && store_tb) store_words(d, d2, tb + i * (NG * WB), kb + i);
                    if (entries && bnd_me && je0 + i >= jlo) store_entry(entry + i);
                }
                continue;
            }
            if (h_state == H_NONE) rebuild_h(k);
            if (h_state == H_LAST) h_from_last();
            h_state = H_ALL;
#pragma unroll 1
            for (; k < kend; ++k) {
                const int r = rs + k;
                uint32_t r0 = __shfl_up_sync(FULL, prmt(X[NP - 1], V[NP - 1], 0x7632), 1);
                uint32_t r1 = __shfl_up_sync(FULL, prmt(X2[NP - 1], sel[C - 1], 0x5432), 1);
                int Hl = __shfl_up_sync(FULL, H[C - 1], 1);
                const uint32_t b0 = __shfl_sync(FULL, bx, k & 31), b1 = __shfl_sync(FULL, by, k & 31);
                const int hb = __shfl_sync(FULL, bh, k & 31);
                if (lane == 0) r0 = b0, r1 = b1, Hl = hb;
#pragma unroll
                for (int c = C - 1; c > 0; --c) sel[c] = sel[c - 1];
                sel[0] = r1 >> 16;
                uint32_t d[NP], d2[NP];
#pragma unroll
                for (int p = 0; p < NP; ++p) d[p] = 0, d2[p] = 0;
                if (r < rlim) {
                    const int st0 = g.st0(r), en0 = g.en0(r);
                    const int st16 = st0 & ~15, en16 = en0 | 15;
                    const int fe = A.generic ? en0 : st0 + ((en0 - st0 + 16) & ~15) - 1;
                    const int before16 = st16 > 0 ? g.st0(r - 1) & ~15 : 0;
                    if (deep && st16 != before16) store_deep(st16);
                    if (col0 == st16 && st16 > 0 && before16 == st16) r0 = prmt(x_in, v_in, 0x5410), r1 = x2_in;
                    uint32_t x = prmt(r0, X[NP - 1], 0x5410), v = prmt(r0, V[NP - 1], 0x5432), x2 = prmt(r1, X2[NP - 1], 0x5410);
                    // score fill
                    const int f0 = st0 - col0, f1 = fe - col0;
                    if (f0 < C && f1 >= 0) {
#pragma unroll
                        for (int p = 0; p < NP; ++p) {
                            const uint32_t m = mask2(p >= f0 && p <= f1, p + NP >= f0 && p + NP <= f1);
                            SS[p] = (score_of(p) & m) | (SS[p] & ~m);
                        }
                    }
                    if (col0 >= st16 && col0 <= en16) {
                        if (r < c0 + SW) {
                            // row 0: the top edge above column r
                            const uint32_t eu = rep2(16 * edge_diff(r, S) + FB);
#pragma unroll
                            for (int p = 0; p < NP; ++p) {
                                const uint32_t m = mask2(col0 + p == r, col0 + p + NP == r);
                                U[p] = (eu & m) | (U[p] & ~m);
                                Y[p] = (K.kxb & m) | (Y[p] & ~m), Y2[p] = (K.kxb2 & m) | (Y2[p] & ~m);
                            }
                        }
#pragma unroll
                        for (int p = NP - 1; p >= 0; --p) {
                            uint32_t xp = p ? X[p - 1] : x, vp = p ? V[p - 1] : v, x2p = p ? X2[p - 1] : x2;
                            cell2<MODE, true>(SS[p], xp, vp, x2p, U[p], Y[p], Y2[p], d[p], K);
                            X[p] = xp, V[p] = vp, X2[p] = x2p;
                            if (MODE == TRACKS) d[p] = vp >> 4, d2[p] = U[p] >> 4;
                        }
                        // H inside the band: on its right edge from the left neighbour, else down
                        const int b0c = st0 - col0, ce = en0 - col0;
                        int hn[C];
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            const int down = H[c] + fval(V[c % NP], c / NP);
                            const int across = (c ? H[c - 1] : Hl) + fval(U[c % NP], c / NP);
                            hn[c] = c == ce ? across : down;
                            hn[c] = c >= b0c && c <= ce ? hn[c] : H[c];
                        }
                        if (en0 == 0 && col0 == 0) hn[0] = r ? H[0] + fval(V[0], 0) : fval(V[0], 0) - S.qe_pre;
#pragma unroll
                        for (int c = 0; c < C; ++c) H[c] = hn[c];
                        if (r >= qm1 || (last_strip && en0 == tm1)) {
                            // end tracking straight into the pair's record (rare cells; the packed
                            // keys make the ">=" later-wins rule an unsigned max, and the strict
                            // earlier-wins rule one on the mirrored position)
                            const int cq = r - qm1 - col0, ctm = tm1 - col0;
#pragma unroll
                            for (int c = 0; c < C; ++c) {
                                if (c < b0c || c > ce) continue;
                                if (c == cq) {
                                    atomicMax(&R->mqe_key, end_key(H[c], pm ^ (col0 + c)));
                                    if (c == ctm) R->score = H[c], R->has_score = 1;
                                }
                                if (c == ctm) {
                                    const unsigned long long key = end_key(H[c], pm ^ (r - tm1));
                                    mte_key = key > mte_key ? key : mte_key;
                                }
                            }
                        }
                    }
                }
                if (STRICT) grown();
                if (CIGAR && store_tb) store_words(d, d2, tb + (k - kb) * (NG * WB), k);
                const int je = r - (c0 + SW - 1);
                if (bnd_me && je >= jlo && je <= jend) store_entry(bnd_me + (je - jlo));
            }
        }
        if (failed) break;
        if (__any_sync(FULL, (int)(peak & 0xffffu) > A.peak_max || (int)(peak >> 16) > A.peak_max) && lane == 0) {
            R->wide = 1;
            atomicExch(A.error + 1, 1);
        }
        if (mte_key && !stopped) atomicMax(&R->mte_key, mte_key);
    }
}

// ---- traceback --------------------------------------------------------------------

struct BtArgs {
    const BandPairDev *pairs;
    int npair;
    const BandStripDev *strips;
    uint8_t *tb;
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
// cell's anti-diagonal (1: deletion, 2: insertion), -1, or -2 for a deep cell whose bytes are not
// computed yet.
template <int WB>
__device__ __forceinline__ int band_force(const Geom &g, const BandStripDev *strips, uint8_t *tb, int i, int j) {
    const int r = i + j, st0 = g.st0(r);
    if (i > (g.en0(r) | 15)) return 1;
    if (i >= (st0 & ~15)) return -1;
    if (i < (st0 & g.bmask)) return 2;
    const int cb = i & g.bmask;
    return *(volatile uint32_t *)DeepRows<WB>::word(tb, strips[cb / SW], cb % SW / C, DeepRows<WB>::WORDS) == 1 ? -1 : -2;
}

// Computes the deep cells of the block that starts at column cb (a warp): the columns below st16
// of its anti-diagonals, from the state each had when st16 passed it, two columns a lane.  Their
// scores stay those of the last fill; column cb takes its left input from column cb + 15 (the
// in-register wrap of the reference's blocks, ksw2_extd2_avx.c:313-330).
template <int WB>
__device__ __noinline__ void deep_fill(const BandPairDev &P, const Geom &g, const BandStripDev &St, uint8_t *tb, int cb,
                                       const KswScore &S, bool right) {
    const int lane = threadIdx.x & 31, B = -g.bmask, lim = min(g.nd, g.rb);
    // the first anti-diagonal whose st0 has reached column X (> 0)
    auto reached = [&](int X) { return min(X + P.qlen - 1, 2 * X + P.w - 1); };
    const int end = min(reached(cb + B), lim);
    int x[2], v[2], x2[2], u[2], y[2], y2[2], s[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) x[c] = v[c] = x2[c] = u[c] = y[c] = y2[c] = s[c] = 0;
    int n = 0;  // columns passed
    for (int r = reached(cb + 16); r < end; ++r) {
        if (n + 16 < B && r == reached(cb + n + 16)) {
            if (2 * lane >= n && 2 * lane < n + 16) {
                // columns 2*lane and 2*lane + 1 of the block: fields of the words of their strip's lane
                const int l = cb % SW / C + lane / 2, f = lane & 1;
                auto at = [&](int w) { return fld(*DeepRows<WB>::word(tb, St, l, w), f); };
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    x[c] = (at(c) - FB) >> 4, v[c] = (at(2 + c) - FB) >> 4, x2[c] = (at(4 + c) - FB) >> 4;
                    u[c] = (at(6 + c) - FB) >> 4, y[c] = (at(8 + c) - FB) >> 4, y2[c] = (at(10 + c) - FB) >> 4;
                    s[c] = (at(12 + c) - 2 * FB) >> 4;
                }
            }
            n += 16;
        }
        int xl = __shfl_up_sync(FULL, x[1], 1), vl = __shfl_up_sync(FULL, v[1], 1), x2l = __shfl_up_sync(FULL, x2[1], 1);
        const int xw = __shfl_sync(FULL, x[1], 7), vw = __shfl_sync(FULL, v[1], 7), x2w = __shfl_sync(FULL, x2[1], 7);
        if (lane == 0) xl = xw, vl = vw, x2l = x2w;
        if (2 * lane >= n) continue;
#pragma unroll
        for (int c = 1; c >= 0; --c) {
            const int xi = c ? x[0] : xl, vi = c ? v[0] : vl, x2i = c ? x2[0] : x2l;
            const int cand[4] = {xi + vi, y[c] + u[c], x2i + vi, y2[c] + u[c]};
            int z = s[c], d = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                // left-aligned: the first candidate wins a tie, right-aligned: the last
                if (right ? cand[k] >= z : cand[k] > z) d = k + 1;
                z = max(z, cand[k]);
            }
            z = min(z, S.mch);
            const int un = z - vi, vn = z - u[c];
            const int open[4] = {cand[0] - z + S.q, cand[1] - z + S.q, cand[2] - z + S.q2, cand[3] - z + S.q2};
#pragma unroll
            for (int k = 0; k < 4; ++k) d |= (right ? open[k] >= 0 : open[k] > 0) ? 8 << k : 0;
            x[c] = max(open[0], 0) - S.qe, y[c] = max(open[1], 0) - S.qe;
            x2[c] = max(open[2], 0) - S.qe2, y2[c] = max(open[3], 0) - S.qe2;
            u[c] = un, v[c] = vn;
            const int t = cb + 2 * lane + c, j = r - t, gr = t % SW / 4;
            if (j < St.jlo || j > St.jend) continue;
            uint8_t *p = tb + St.tb_off + ((int64_t)(j - St.jlo + 4 * gr) * NG + gr) * WB + t % 4;
            if (WB == 8) p[0] = (uint8_t)vn, p[4] = (uint8_t)un;
            else p[0] = (uint8_t)d;
        }
    }
    __syncwarp();
    if (lane == 0) *DeepRows<WB>::word(tb, St, cb % SW / C, DeepRows<WB>::WORDS) = 1;
    __threadfence_block();
    __syncwarp();
}

// The stored rows of a column group (4 columns) of a pair's strips (words of WB bytes).
template <int WB>
__device__ __forceinline__ TbGroup band_group(const BandStripDev *strips, const uint8_t *tb, int tlen, int col_lo,
                                              int gg) {
    if (gg < 0 || gg * 4 >= tlen || gg * 4 < col_lo) return TbGroup{tb, 0, -1};
    const BandStripDev St = strips[gg / NG];
    const int g = gg % NG;
    return TbGroup{tb + St.tb_off + ((int64_t)4 * g * NG + g) * WB, St.jlo, St.jend};
}

// Warps per block of the finishing kernel: the Singletrack words are twice as large, and its
// gap search has two tiles of its own.
template <bool ST>
constexpr int fin_warps() { return ST ? 1 : 4; }

// Result record of one pair, then ksw_backtrack (minimap2/ksw2.h:160-192) with the
// off/off_end forcing of the band, or the Singletrack reconstruction
// (minimap2/ksw2_singletrack.cpp:63-176); one warp per pair walks in runs (tb_walk.cuh).
template <bool ST>
__global__ void __launch_bounds__(32 * fin_warps<ST>()) ksw_band_finish_kernel(BtArgs A) {
    constexpr int WB = ST ? 8 : 4;
    using Window = TbWindow<WB, 4, ST ? 1 : 0, true>;
    using Probe = TbWindow<WB, 4, 0, false>;  // the rows and columns of a Singletrack gap search
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
    uint8_t *tb = A.tb;
    auto force = [&](int a, int b) { return band_force<WB>(g, strips, tb, a, b); };
    auto fill = [&](int a, int) {
        deep_fill<WB>(P, g, strips[a / SW], tb, a & g.bmask, A.sc, (flag & AW_EZ_RIGHT) != 0);
    };
    Window win;
    win.init(tiles[warp], NG * WB);
    auto grp = [&](int gg) -> TbGroup { return band_group<WB>(strips, tb, tlen, 0, gg); };
    WarpCigar cg{A.cig + P.cig_off, 0, 0, 0};
    if (cigar && ST) {
        // ksw_extd2_singletrack_sse reconstructs whatever the EXTZ/SEMIGLOBAL flags
        // (minimap2/ksw2_singletrack.cpp:606-615)
        if (!o.zdropped && (sse_st || !(flag & (AW_EZ_EXTZ_ONLY | AW_EZ_SEMIGLOBAL_END)))) {
            const uint8_t *qs = A.qcodes + P.qoff, *ts = A.tcodes + P.toff;
            Probe probe;
            probe.init(tiles[warp] + Window::BYTES, NG * WB);
            int i = tlen - 1, j = qlen - 1;
            if (tb_singletrack(i, j, cg, win, probe, grp, force, fill, A.sc, A.mat, A.m, qs, ts)) {
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
            tb_walk(i, j, state, 0, cg, win, grp, force, fill);
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
__global__ void __launch_bounds__(32) ksw_band_round_walk_kernel(BtArgs A, const BandGroupDev *groups) {
    using Window = TbWindow<4, 4, 0, true>;
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
    uint8_t *tb = A.tb;
    Window win;
    win.init(tiles, NG * 4);
    auto grp = [&](int gg) -> TbGroup { return band_group<4>(strips, tb, tlen, col_lo, gg); };
    WarpCigar cg{A.cig + P.cig_off, w.n, (uint32_t)w.op, w.len};
    int i = w.i, j = w.j, state = w.state;
    tb_walk(i, j, state, col_lo, cg, win, grp, [&](int a, int b) { return band_force<4>(g, strips, tb, a, b); },
            [&](int a, int) { deep_fill<4>(P, g, strips[a / SW], tb, a & g.bmask, A.sc, (A.flag & AW_EZ_RIGHT) != 0); });
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

typedef void (*BandKernel)(BandArgs);
template <bool STRICT>
BandKernel band_kernel_of(int flag, int block) {
    if (flag & AW_EZ_SCORE_ONLY) return ksw_band_kernel<SCORES, STRICT>;
    if (singletrack_tracks(flag, block)) return ksw_band_kernel<TRACKS, STRICT>;
    return (flag & AW_EZ_RIGHT) ? ksw_band_kernel<RIGHTMOST, STRICT> : ksw_band_kernel<LEFT, STRICT>;
}
BandKernel band_kernel_for(int flag, int block, bool strict) {
    return strict ? band_kernel_of<true>(flag, block) : band_kernel_of<false>(flag, block);
}

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// x, y, x2 and y2 grow by grow = M - min(e, e2) a step at most, and a candidate adds a u or v of at
// most M (ksw2_cell.cuh).  Within 30 steps at the band's left edge (16 columns) they reach 30 * grow: 149 under (4, 2,
// 24, 1), 989 under (30, 4, 40, 1); in the band and above it 57 was the largest value met.  A look
// every PUB steps has room for that while grow is below 39; above, every step is checked (and a gap
// that costs 49 to open still sends some pairs to the anti-diagonal kernel).
int band_uv(const KswScore &S) { return std::max(S.qe, -S.long_diff); }  // M
int band_grow(const KswScore &S) { return band_uv(S) - std::min(S.e, S.e2); }
bool band_strict(const KswScore &S) { return 30 * band_grow(S) + 57 > CAND_MAX - band_uv(S) - PUB * band_grow(S); }
int band_peak_max(const KswScore &S) {
    return 16 * std::max(CAND_MAX - band_uv(S) - (band_strict(S) ? 1 : PUB) * band_grow(S), 0) + FB;
}

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
                    int flag, int block, int64_t tb_budget, std::vector<int32_t> *refused) {
    bp = BandPlan();
    bp.block = block;
    const bool cigar = !(flag & AW_EZ_SCORE_ONLY);
    const bool st = cigar && singletrack_tracks(flag, block);
    const int WB = st ? 8 : 4;  // bytes of a traceback word
    const int B = block;
    struct PairGeo {
        int32_t id, ww, rb;
        int64_t tb, bnd;
        int64_t tail;  // bytes by which the skew of its strips reaches beyond their rows (<= 32 KB)
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
        const int nstrip = (int)ceil_div(tl, SW), deep_rows = deep_cells(B, ww, ql) ? 64 / WB : 0;
        G.tb = 0, G.bnd = 0, G.tail = 0;
        int64_t reach = 0;
        for (int s = 0; s < nstrip; ++s) {
            const int c0 = s * SW;
            BandStripDev sd;
            // the strip's first anti-diagonal: the score fill reaches its first column (15 past
            // en0 at most); jstart is the row of that column there
            sd.jstart = (int)(std::max<int64_t>(std::max<int64_t>(0, c0 - 15), 2 * ((int64_t)c0 - 15) - ww) - c0);
            // stored rows: from the first row of any of its columns that may be computed (no
            // earlier than c0-w-32) to the last one that is (stB <= t)
            sd.jlo = (int)std::max<int64_t>(0, (int64_t)c0 - ww - 32);
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
                if (cigar) {
                    stb = (rows + deep_rows) * NG * WB;
                    reach = std::max(reach, G.tb + stb + 4 * (ceil_div(std::min(SW, tl - c0), 4) - 1) * NG * WB);
                }
                G.tb += stb;
                if (s + 1 < nstrip) G.bnd += rows;  // the last strip's column is not read
            }
            G.stb.push_back(stb);
            G.strips.push_back(sd);
            G.start.push_back((int64_t)sd.jstart + c0);  // its first step
        }
        G.tail = (std::max(reach, G.tb) - G.tb + 255) / 256 * 256;
        G.tb = (G.tb + 255) / 256 * 256;
        if (G.rb < nd) {
            // the band becomes empty before the end: the reference stops there with
            // zdropped = 1 and no traceback (ksw2_extd2_sse.c:151-154), so the DP runs without
            // storing one (the first pass of a recomputed pair, with nothing to recompute)
            G.ckpt = G.notb = true;
            G.tb = G.tail = 0;
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
    // What a pair alone may take: the tail is not charged, and of the boundary columns only as many
    // as strips of twice the width would have, so that the narrow strips refuse nothing that wider
    // ones would run (the two arenas then exceed the budget by 1/64 of the traceback at most).
    const int64_t cap_one = std::max<int64_t>(tb_budget - std::min(bnd_all / 2, tb_budget / 3), 1);
    for (PairGeo &G : geo) {
        if (G.notb) continue;
        // Singletrack pairs keep their whole two-track traceback: the reconstruction probes
        // arbitrarily far left in one gap search, so it cannot be split into strip groups.  A
        // pair whose traceback does not fit is refused like an allocation failure of the
        // reference (ksw2_extd2_avx.c:206-210: reset result, zdropped = 1).
        bool refuse = st && G.tb > cap_one;
        if (!st && G.tb + G.tail > cap_tb) {
            // Traceback beyond the budget: the first pass stores only the strips' boundary
            // columns; then the traceback is recomputed in groups of strips, from the last group
            // to the first, each from the stored column on its left, and the walk continues
            // through each group as it is recomputed.  The groups are cut per wave (below).
            for (int s = 0; s < (int)G.strips.size(); ++s) refuse |= G.stb[s] > cap_one;
            if (!refuse) {
                G.ckpt = true;
                G.tb = G.tail = 0;  // the first pass stores no traceback
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
        bp.tb_total += G.tb + G.tail;
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
        const int64_t pb = band_bnd_bytes(G.bnd), ptb = G.tb + G.tail;
        int best = -1;
        for (size_t k = 0; k < wv.size(); ++k) {
            if (wtb[k] + ptb <= cap_tb && wbnd[k] + pb <= cap_bnd &&
                (best < 0 || wbnd[k] * cap_tb + wtb[k] * cap_bnd < wbnd[best] * cap_tb + wtb[best] * cap_bnd))
                best = (int)k;
        }
        if (best < 0) {
            wv.emplace_back();
            wtb.push_back(0), wbnd.push_back(0);
            best = (int)wv.size() - 1;
        }
        wtb[best] += ptb, wbnd[best] += pb;
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
            tb += G.tb + G.tail;
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
            const int64_t tail = 4 * (NG - 1) * NG * WB;
            const int64_t share = std::max<int64_t>((int64_t)((double)gres * tb_pair / std::max(tb_all, 1.0)) - tail, 1);
            int s1 = (int)G.strips.size();
            while (s1 > 0) {
                int s0 = s1 - 1;
                int64_t acc = G.stb[s0];
                while (s0 > 0 && acc + G.stb[s0 - 1] <= share) acc += G.stb[--s0];
                groups[c].push_back({s0, s1});
                gtb[c].push_back(acc + tail);
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

int band_occupancy(int flag, int block) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, band_kernel_for(flag, block, false), 32 * BAND_WARPS, 0) != cudaSuccess)
        return 1;
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
    a.peak_max = band_peak_max(S);
    return band_launch_units(bp, a, flag, ctas, st);
}

cudaError_t band_launch_units(const BandPlan &bp, const BandArgs &a, int flag, int ctas, cudaStream_t st) {
    const int grid = std::max(1, std::min(ctas, (a.n_units + BAND_WARPS - 1) / BAND_WARPS));
    band_kernel_for(flag, bp.block, band_strict(a.sc))<<<grid, 32 * BAND_WARPS, 0, st>>>(a);
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
    if (stk) ksw_band_finish_kernel<true><<<grid, 32 * fw, 0, st>>>(b);
    else ksw_band_finish_kernel<false><<<grid, 32 * fw, 0, st>>>(b);
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
        a.peak_max = band_peak_max(S);
        if ((e = band_launch_units(bp, a, flag, ctas, st)) != cudaSuccess) return e;
        ksw_band_round_walk_kernel<<<R.ngroup, 32, 0, st>>>(b, gd);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace aw
