// KSW2 extd2, full-matrix form (w < 0 or w >= max(qlen, tlen)), on sm_100a.
//
// Same recurrence as minimap2/ksw2_extd2_sse.c:43-71 + :237-330 (difference-
// encoded u, v, x, y, x2, y2 cells; state byte d with the 3-bit argmax and the
// four continuation bits).  In full mode every cell the recurrence reads is a real
// matrix cell or a matrix edge, so the SIMD padding lanes of the reference never
// influence the result and are not computed here.  The host only routes parameter
// sets to this kernel whose int8 intermediates provably cannot wrap
// (ksw2_api.cu: full_path_ok).
//
// Two cells per instruction.  Every register holds two 16-bit fields, each a cell
// value stored as 16*value + bias; the two fields are cells of two different rows
// (below), so a cell is DPX SIMD (vimax3 / viaddmin .s16x2, vmax / vmin .s16x2) plus
// 32-bit adds whose per-field results stay inside [0, 65536), which the biases
// guarantee, so no carry crosses from one field into the other.  The low 4 bits of a
// field are free: the five candidates of the max carry a priority tag there, so one
// max yields both z and the arg-max under the reference's tie rule (left-aligned: the
// first candidate wins a tie, ksw2_extd2_sse.c:244-251; right-aligned: the last,
// :291-298).
//
// Work decomposition:
//   * target columns are cut into strips of 32 lanes x 2*NP columns; lane L owns NP columns in
//     its low fields and the next NP in its high fields.  NP = 8 (strips of 512 columns) does
//     the most cells per step; NP = 2 (strips of 128) has the shortest step, for pairs whose
//     chain of steps would be longer than the batch (one 5 kb pair: 4.1 -> 1.3 ms);
//   * a warp sweeps the query rows of its strip with a skew of two steps per lane and
//     one step between the halves: at step k lane L computes row k-2L in its low fields
//     and row k-2L-1 in its high fields, so the (x, v, x2) of its last low column feed its
//     first high column at the next step, and its last high column reaches lane L+1 by one
//     __shfl_up per step; the query code travels one step ahead of its row, so the score
//     loads do not wait for the shuffle;
//   * strip s+1 takes its left edge (the last column of strip s) from a global boundary
//     buffer that strip s fills row by row.  An entry carries a written mark (the buffer is
//     zero before the launch), and a strip reads eight rows ahead, so neither side needs a
//     fence or a counter and a pair's strips run on any warps of the grid;
//   * units of work come from a device queue (atomicAdd on a head counter), largest pairs
//     first: the strips of a pair one by one, left to right (a strip only ever waits for a
//     unit that was taken before it), or a whole pair, whose strips one warp then sweeps one
//     after the other without waiting;
//   * the traceback bytes of a step go to HBM as one coalesced store per warp, with
//     evict-first policy (they are read back along one path);
//   * H is not carried per cell: the last row's H (mqe, the score) is a prefix sum of
//     the last row's u along the strip after the sweep, and the last column's H (mte)
//     is accumulated by the lane that owns that column.
// The Singletrack traceback (minimap2/ksw2_singletrack.cpp) keeps v and u of every cell
// instead of the state byte; in full mode its cells are the same.
#include "aw_internal.h"
#include "ksw2_cell.cuh"
#include "tb_walk.cuh"
#include <atomic>
#include <climits>
#include <cstring>
#include <type_traits>

namespace aw {

namespace {

constexpr unsigned FULLMASK = 0xffffffffu;

// H(t, -1) (= H(-1, t)): sum of edge_diff(0..t), the score of a leading gap of length
// t+1, offset as the reference's H[0] = v[0] - qe with qe taken before the swap.
__device__ __forceinline__ int htop(int t, const KswScore &S) {
    const int L = S.long_thres;
    int A = min(t, L - 1);
    A = A < 0 ? 0 : A;
    const int eq = (L >= 1 && L <= t) ? 1 : 0;
    const int B = t - A - eq;
    // the reference seeds H[0] with the pre-swap q+e, which shifts every H equally
    return -S.qe_pre - A * S.e + eq * S.long_diff - B * S.e2;
}

// Lexicographic (value, position) maximum: later positions win ties, the
// ">=" end-tracking rule of ksw2_extd2_sse.c:369-372.
__device__ __forceinline__ void best_merge(int &v, int &p, int ov, int op) {
    if (ov > v || (ov == v && op > p)) v = ov, p = op;
}

// Score profile of a lane: for each query code q (0..7) the tagged score fields of the lane's
// columns, in shared memory, read back by the same lane only.  NP = 8: two vectors of 16 B
// (low and high columns) per lane and code; lanes with bit 2 set store them swapped, so the 8
// lanes of a quarter-warp load 16 B each from distinct banks.  NP = 2: one word each, the
// low columns' words of a warp together, then the high columns'.
template <int NP>
struct Prof {
    static constexpr int CODE = 32 * 4 * NP;  // bytes per code (one warp)
    static constexpr int WARP = 8 * CODE;     // bytes per warp
    using Vec = typename std::conditional<NP == 8, uint4, uint32_t>::type;
    static __device__ __forceinline__ int lo(int lane) { return NP == 8 ? lane * 32 + 16 * ((lane >> 2) & 1) : lane * 4; }
    static __device__ __forceinline__ int hi(int lane) {
        return NP == 8 ? lane * 32 + 16 * (1 - ((lane >> 2) & 1)) : 128 + lane * 4;
    }
};
__device__ __forceinline__ uint32_t vword(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
__device__ __forceinline__ uint32_t vword(const uint32_t &v, int) { return v; }

// State of one warp's sweep over one strip.
template <int NP>
struct Sweep {
    uint32_t U[NP], Y[NP], Y2[NP];  // column state, column pair c = (col0 + c, col0 + NP + c)
    uint32_t X, V, X2;              // values flowing right; after a step: the outputs of the last column pair
    uint32_t qlo, qhi;              // query codes of the rows of the low / high fields at the next step
    uint32_t vcap;                  // last strip: v of the pair's last column at the last step
    uint32_t held, held2;           // NP = 2: the low columns' traceback bytes (and u bytes) of the last step
};

// Boundary entries: x | v << 16, x2 | mark << 16; the last row's H and the mark.
constexpr uint32_t BND_MARK = 0x80000000u;
__device__ __forceinline__ uint2 bnd_load(const uint2 *p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return make_uint2((uint32_t)v, (uint32_t)(v >> 32));
}
__device__ __forceinline__ void bnd_store(uint2 *p, uint32_t x, uint32_t y) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((uint64_t)(y | BND_MARK) << 32 | x) : "memory");
}

// Per-strip context shared by the steps.
struct StripCtx {
    int qlen, lane, c_lane, c_fld, c_cc;
    uint2 *bnd;                 // this strip's boundary column; null: no right neighbour, or not this lane
    const uint8_t *prof_lo, *prof_hi;
    uint8_t *tb;                // this lane's traceback word of step 0 of the strip
};

// The bytes 0..NP-1 of the low fields in the low half's words and those of the high fields
// in the high half's, from one byte per field (bits 0-7 and 16-23 of each t).
template <int NP>
struct Packed {
    uint32_t lo[NP / 4 + (NP < 4)], hi[NP / 4 + (NP < 4)];
};
__device__ __forceinline__ uint32_t two(uint32_t a, uint32_t b) { return prmt(a, b, 0x6240); }
__device__ __forceinline__ Packed<8> pack(const uint32_t (&t)[8]) {
    const uint32_t a = two(t[0], t[1]), b = two(t[2], t[3]), c = two(t[4], t[5]), d = two(t[6], t[7]);
    return Packed<8>{{prmt(a, b, 0x5410), prmt(c, d, 0x5410)}, {prmt(a, b, 0x7632), prmt(c, d, 0x7632)}};
}
__device__ __forceinline__ Packed<2> pack(const uint32_t (&t)[2]) {
    const uint32_t a = two(t[0], t[1]);
    return Packed<2>{{a & 0xffffu}, {a >> 16}};
}

// Traceback bytes of a lane-step.
template <int MODE, int NP>
constexpr int word_bytes() { return MODE == SCORES ? 0 : 2 * NP * (MODE == TRACKS ? 2 : 1); }

// Steps [k0, k1) of a strip (at most 8); bx/by: lane i holds the left values of lane 0 for row
// (k0 & ~31) + i, with the query code of the row after it in by's high half.  At step k the
// low fields are row jlo = k - 2*lane and the high fields row jlo - 1; the high fields take the
// low fields' last column of the previous step.  MASKED: some field of the warp may be outside
// [0, qlen): those fields start from safe left values and keep their column state.  LAST:
// the strip holds the pair's last column.
template <int MODE, int NP, bool MASKED, bool LAST>
__device__ __forceinline__ void sweep_steps(Sweep<NP> &w, const StripCtx &C, int k0, int k1, uint32_t bx, uint32_t by,
                                            const CellK &K, int &hm16, int &mte16, int &mte_q) {
    using P = Prof<NP>;
    constexpr int WORD = word_bytes<MODE, NP>();
    typename P::Vec nlo, nhi;
    if (NP == 2) {
        nlo = *reinterpret_cast<const typename P::Vec *>(C.prof_lo + w.qlo * P::CODE);
        nhi = *reinterpret_cast<const typename P::Vec *>(C.prof_hi + w.qhi * P::CODE);
    }
    uint8_t *tb = C.tb + (int64_t)k0 * (32 * WORD);
    uint2 *bnd = C.bnd + (k0 - KSW_LAG);  // the row of lane 31's high fields
#pragma unroll 1
    for (int k = k0; k < k1; ++k, tb += 32 * WORD, ++bnd) {
        const uint32_t w0 = prmt(w.X, w.V, 0x7632), w1 = prmt(w.X2, w.qhi, 0x5432);
        uint32_t r0 = __shfl_up_sync(FULLMASK, w0, 1), r1 = __shfl_up_sync(FULLMASK, w1, 1);
        const uint32_t b0 = __shfl_sync(FULLMASK, bx, k & 31), b1 = __shfl_sync(FULLMASK, by, k & 31);
        typename P::Vec slo, shi;
        if (NP == 2) {
            slo = nlo, shi = nhi;
        } else {
            slo = *reinterpret_cast<const typename P::Vec *>(C.prof_lo + w.qlo * P::CODE);
            shi = *reinterpret_cast<const typename P::Vec *>(C.prof_hi + w.qhi * P::CODE);
        }
        if (C.lane == 0) r0 = b0, r1 = b1;
        const int jlo = k - 2 * C.lane;
        uint32_t X = prmt(r0, w.X, 0x5410), V = prmt(r0, w.V, 0x5432), X2 = prmt(r1, w.X2, 0x5410);
        w.qhi = w.qlo, w.qlo = r1 >> 16;  // the codes of the next step
        if (NP == 2) {
            nlo = *reinterpret_cast<const typename P::Vec *>(C.prof_lo + w.qlo * P::CODE);
            nhi = *reinterpret_cast<const typename P::Vec *>(C.prof_hi + w.qhi * P::CODE);
        }
        uint32_t M = 0xffffffffu;
        if (MASKED) {
            M = ((unsigned)jlo < (unsigned)C.qlen ? 0x0000ffffu : 0u) |
                ((unsigned)(jlo - 1) < (unsigned)C.qlen ? 0xffff0000u : 0u);
            X = (X & M) | (K.kxa & ~M);
            V = (V & M) | (rep2(FB) & ~M);
            X2 = (X2 & M) | (K.kxa2 & ~M);
        }
        uint32_t D[NP], D2[NP];
#pragma unroll
        for (int c = 0; c < NP; ++c) {
            const uint32_t sc = prmt(vword(slo, c >> 1), vword(shi, c >> 1), (c & 1) ? 0x7632 : 0x5410);
            uint32_t u = w.U[c], y = w.Y[c], y2 = w.Y2[c];
            cell2<MODE, NP == 2>(sc, X, V, X2, u, y, y2, D[c], K);
            // a field's byte of 16 * value + FB, shifted down by 4: the value (FB is a multiple of 16 * 256)
            if (MODE == TRACKS) D[c] = V >> 4, D2[c] = u >> 4;
            if (MASKED) {
                w.U[c] = (u & M) | (w.U[c] & ~M);
                w.Y[c] = (y & M) | (w.Y[c] & ~M);
                w.Y2[c] = (y2 & M) | (w.Y2[c] & ~M);
            } else {
                w.U[c] = u, w.Y[c] = y, w.Y2[c] = y2;
            }
            if (LAST && c == C.c_cc) w.vcap = V;
        }
        w.X = X, w.V = V, w.X2 = X2;
        if constexpr (MODE != SCORES) {
            const auto d = pack(D);
            if constexpr (NP == 8) {
                uint4 *dst = reinterpret_cast<uint4 *>(tb);
                if constexpr (MODE == TRACKS) {
                    const auto e = pack(D2);
                    __stcs(dst, make_uint4(d.lo[0], d.lo[1], e.lo[0], e.lo[1]));
                    __stcs(dst + 1, make_uint4(d.hi[0], d.hi[1], e.hi[0], e.hi[1]));
                } else {
                    __stcs(dst, make_uint4(d.lo[0], d.lo[1], d.hi[0], d.hi[1]));
                }
            } else {
                // the row of the high fields: its low columns were computed at the last step
                if constexpr (MODE == TRACKS) {
                    const auto e = pack(D2);
                    __stcs(reinterpret_cast<uint2 *>(tb), make_uint2(w.held | d.hi[0] << 16, w.held2 | e.hi[0] << 16));
                    w.held2 = e.lo[0];
                } else {
                    __stcs(reinterpret_cast<uint32_t *>(tb), w.held | d.hi[0] << 16);
                }
                w.held = d.lo[0];
            }
        }
        if (LAST && C.lane == C.c_lane) {
            const int row = jlo - C.c_fld;
            if ((unsigned)row < (unsigned)C.qlen) {
                hm16 += fld(w.vcap, C.c_fld) - FB;
                if (hm16 >= mte16) mte16 = hm16, mte_q = row;
            }
        }
        // lane 31 of a strip with a right neighbour
        if (C.bnd && (!MASKED || k >= KSW_LAG)) bnd_store(bnd, prmt(w.X, w.V, 0x7632), w.X2 >> 16);
    }
}

__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr uint64_t WAIT_NS = 20ull * 1000 * 1000 * 1000;  // bounded wait on the left strip
constexpr int GROUP = 8;  // steps between two looks at the left column

__device__ __forceinline__ unsigned long long mqe_key(int v, int pos) {
    return ((unsigned long long)((uint32_t)v ^ 0x80000000u) << 32) | (uint32_t)pos;
}

// Warps per CTA: a wide strip's warps hide one another's latencies; narrow strips are few and
// latency-bound, and small CTAs spread them over the SMs.
template <int NP>
constexpr int cta_warps() { return NP == 8 ? 8 : 4; }

template <int MODE, int NP>
__global__ void __launch_bounds__(32 * cta_warps<NP>(), NP == 8 ? 2 : 5) ksw_full_kernel(KswFullArgs A) {
    extern __shared__ __align__(16) uint8_t prof_smem[];
    using PF = Prof<NP>;
    using T = Tags<MODE>;
    constexpr int COLS = 2 * NP, STRIP = 32 * COLS;
    constexpr int WORD = word_bytes<MODE, NP>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const KswScore &S = A.sc;
    const CellK K = make_cellk<MODE>(S, A.one);
    uint8_t *prof = prof_smem + warp * PF::WARP;

    for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(A.queue, 1);
        u = __shfl_sync(FULLMASK, u, 0);
        if (u >= A.n) break;
        const int2 un = A.units ? A.units[u] : make_int2(0, u);
        const int idx = un.x;
        const KswPair P = A.pairs[idx];
        const int qlen = P.qlen, tlen = P.tlen, tl1 = tlen - 1;
        const uint8_t *qs = A.qcodes + P.qoff, *ts = A.tcodes + P.toff;
        const int nstrip = (tlen + STRIP - 1) / STRIP;
        volatile int32_t *stop_word = &A.res[idx].stopped;
        uint2 *bnd = reinterpret_cast<uint2 *>(A.bnd + P.bnd_off);
        StripCtx C;
        C.qlen = qlen, C.lane = lane;
        C.prof_lo = prof + PF::lo(lane), C.prof_hi = prof + PF::hi(lane);
        // the pair's last column: owning lane, field and column pair (in the last strip)
        C.c_lane = tl1 % STRIP / COLS, C.c_fld = tl1 / NP & 1, C.c_cc = tl1 % NP;
        bool stopped = false, failed = false;
        const int s_end = un.y < 0 ? nstrip : un.y + 1;
        for (int s = un.y < 0 ? 0 : un.y; s < s_end && !stopped && !failed; ++s) {
            const int col0 = s * STRIP + lane * COLS;
            const bool last = s == nstrip - 1;
            // boundary column of strip s: rows at [s * (qlen + 1), +qlen), its last-row H after them
            const uint2 *left = s > 0 ? bnd + (int64_t)(s - 1) * (qlen + 1) : nullptr;
            uint2 *mine = last ? nullptr : bnd + (int64_t)s * (qlen + 1);
            C.bnd = lane == 31 ? mine : nullptr;
            C.tb = MODE != SCORES ? A.tb + P.tb_off + ((int64_t)s * (qlen + KSW_LAG) * 32 + lane) * WORD : nullptr;
            // score profile of the lane's columns for query codes 0..7
            {
                uint32_t tlo[COLS], thi[COLS];
#pragma unroll
                for (int c = 0; c < COLS; ++c) {
                    const int col = col0 + c;
                    const int tc = col < tlen ? (ts[col] & 7) : 0;
                    tlo[c] = S.tab_lo[tc], thi[c] = S.tab_hi[tc];
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    uint32_t wd[NP];
#pragma unroll
                    for (int i = 0; i < NP; ++i) {
                        const int sa = (int)(int8_t)(uint8_t)(((q < 4 ? tlo[2 * i] : thi[2 * i]) >> (8 * (q & 3))) & 0xff);
                        const int sb =
                            (int)(int8_t)(uint8_t)(((q < 4 ? tlo[2 * i + 1] : thi[2 * i + 1]) >> (8 * (q & 3))) & 0xff);
                        wd[i] = (uint32_t)(16 * sa + T::s + 2 * FB) | ((uint32_t)(16 * sb + T::s + 2 * FB) << 16);
                    }
                    if constexpr (NP == 8) {
                        *reinterpret_cast<uint4 *>(prof + PF::lo(lane) + q * PF::CODE) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
                        *reinterpret_cast<uint4 *>(prof + PF::hi(lane) + q * PF::CODE) = make_uint4(wd[4], wd[5], wd[6], wd[7]);
                    } else {
                        *reinterpret_cast<uint32_t *>(prof + PF::lo(lane) + q * PF::CODE) = wd[0];
                        *reinterpret_cast<uint32_t *>(prof + PF::hi(lane) + q * PF::CODE) = wd[1];
                    }
                }
            }
            Sweep<NP> w;
#pragma unroll
            for (int c = 0; c < NP; ++c) {
                w.U[c] = (uint32_t)(16 * edge_diff(col0 + c, S) + FB) |
                         ((uint32_t)(16 * edge_diff(col0 + NP + c, S) + FB) << 16);
                w.Y[c] = K.kxb;
                w.Y2[c] = K.kxb2;
            }
            w.X = K.kxa, w.V = rep2(FB), w.X2 = K.kxa2;
            w.qlo = lane == 0 ? qs[0] & 7u : 0u, w.qhi = 0, w.vcap = rep2(FB), w.held = w.held2 = 0;
            int hm16 = 16 * htop(tl1, S);  // H(-1, tlen-1), then down the last column
            int mte16 = INT_MIN, mte_q = -1;
            const uint32_t edge_x = K.kxa & 0xffffu, edge_x2 = K.kxa2 & 0xffffu;
            // lane 0's left values of a row, marked; rows past the last need none
            auto left_of = [&](int row) -> uint2 {
                if (row >= qlen) return make_uint2(0u, BND_MARK);
                if (s == 0) return make_uint2(edge_x | ((uint32_t)(16 * edge_diff(row, S) + FB) << 16), edge_x2 | BND_MARK);
                return bnd_load(left + row);
            };
            // waits (bounded) until every lane with want has its entry
            auto await = [&](uint2 &e, bool want, auto &&load) {
                if (__all_sync(FULLMASK, !want || (e.y & BND_MARK))) return;
                const uint64_t t0 = globaltimer();
                unsigned ns = 16, polls = 0;
                for (;;) {
                    if (want && !(e.y & BND_MARK)) e = load();
                    if (__all_sync(FULLMASK, !want || (e.y & BND_MARK))) return;
                    if (A.deadline && __shfl_sync(FULLMASK, lane == 0 ? *stop_word : 0, 0)) {
                        stopped = true;  // the strip on the left stopped at the deadline
                        return;
                    }
                    // the bound and the error flag (another warp gave up), every 32 polls
                    if ((++polls & 31) == 0 &&
                        __any_sync(FULLMASK, globaltimer() - t0 > WAIT_NS || *(volatile int32_t *)A.error)) {
                        failed = true;
                        if (lane == 0) atomicExch(A.error, 1);
                        return;
                    }
                    __nanosleep(ns);
                    ns = ns < 256 ? ns * 2 : ns;
                }
            };
            // past the deadline: no score and no traceback (ksw2_extd2_sse.c:136-139, :400-409), and
            // the ends as far as the pair got.  Its last strip always comes here, as it cannot
            // finish without those on its left; the warp of a whole pair may stop before it.
            auto report_stop = [&]() {
                if (lane != C.c_lane || (!last && un.y >= 0)) return;
                const unsigned long long k = *(volatile unsigned long long *)&A.res[idx].mqe_key;
                KswOut o;
                o.score = AW_NEG_INF, o.max = 0, o.max_q = -1, o.max_t = -1;
                o.mqe = k ? (int)((uint32_t)(k >> 32) ^ 0x80000000u) : AW_NEG_INF, o.mqe_t = k ? (int)(uint32_t)k : -1;
                o.mte = last && mte_q >= 0 ? mte16 >> 4 : AW_NEG_INF, o.mte_q = last ? mte_q : -1;
                o.n_cigar = 0, o.zdropped = 0, o.reach_end = 0, o.stopped = 1;
                A.out[idx] = o;
            };
            auto code_of = [&](int row) -> uint32_t { return row < qlen ? (qs[row] & 7u) << 16 : 0u; };
            // lane i holds what lane 0 needs for row (k & ~31) + i: the next group's entries and
            // the next 32 query codes are on their way while the current ones are used
            uint2 ahead = make_uint2(0u, BND_MARK);
            if (lane < GROUP) ahead = left_of(lane);
            uint32_t qnext = code_of(lane + 1), qcur = 0, bx = 0, by = 0;
            const int last_k = qlen + KSW_LAG;
            for (int k0 = 0; k0 < last_k; k0 += GROUP) {
                if ((k0 & 31) == 0) {
                    if (A.deadline) {
                        // cooperative stop, polled every 32 rows (ksw2_progress.c:30-38 polls
                        // every 256 anti-diagonals); any strip stops the pair
                        int st = 0;
                        if (lane == 0) {
                            st = *stop_word;
                            if (!st && aw_deadline_passed(A.deadline)) st = 1, atomicExch((int32_t *)stop_word, 1);
                        }
                        if (__shfl_sync(FULLMASK, st, 0)) {
                            stopped = true;
                            break;
                        }
                    }
                    qcur = qnext;
                    qnext = code_of(k0 + 32 + lane + 1);
                }
                const bool now = (lane & ~(GROUP - 1)) == (k0 & 31);
                await(ahead, now, [&]() { return left_of((k0 & ~31) + lane); });
                if (stopped || failed) break;
                if (now) bx = ahead.x, by = (ahead.y & 0xffffu) | qcur;
                if ((lane & ~(GROUP - 1)) == ((k0 + GROUP) & 31)) ahead = left_of(((k0 + GROUP) & ~31) + lane);
                const int k1 = min(k0 + GROUP, last_k);
                // every field of every lane is inside [0, qlen) for k in [KSW_LAG, qlen)
                if (k0 >= KSW_LAG && k1 <= qlen) {
                    if (last) sweep_steps<MODE, NP, false, true>(w, C, k0, k1, bx, by, K, hm16, mte16, mte_q);
                    else sweep_steps<MODE, NP, false, false>(w, C, k0, k1, bx, by, K, hm16, mte16, mte_q);
                } else {
                    if (last) sweep_steps<MODE, NP, true, true>(w, C, k0, k1, bx, by, K, hm16, mte16, mte_q);
                    else sweep_steps<MODE, NP, true, false>(w, C, k0, k1, bx, by, K, hm16, mte16, mte_q);
                }
            }
            __syncwarp();
            if (stopped) report_stop();
            if (stopped || failed) break;
            // last row: H(qlen-1, col) = H(qlen-1, col0 - 1) + the prefix sum of the last
            // row's u (the column state after the sweep) along the strip
            int lsum = 0;
#pragma unroll
            for (int c = 0; c < NP; ++c) lsum += fld(w.U[c], 0) + fld(w.U[c], 1) - 2 * FB;
            int incl = lsum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULLMASK, incl, o);
                if (lane >= o) incl += t;
            }
            int base16 = 16 * htop(qlen - 1, S);
            if (s > 0) {
                uint2 e = lane == 0 ? bnd_load(left + qlen) : make_uint2(0u, 0u);
                await(e, lane == 0, [&]() { return bnd_load(left + qlen); });
                if (stopped) report_stop();
                if (stopped || failed) break;
                __threadfence();  // what the strips on the left put into the pair's record before it
                base16 = (int)__shfl_sync(FULLMASK, e.x, 0);
            }
            int h = base16 + incl - lsum, mqe16 = INT_MIN, mqe_t = -1, score16 = INT_MIN;
#pragma unroll
            for (int f = 0; f < 2; ++f) {
#pragma unroll
                for (int c = 0; c < NP; ++c) {
                    h += fld(w.U[c], f) - FB;
                    const int col = col0 + NP * f + c;
                    if (col < tlen) {
                        if (h >= mqe16) mqe16 = h, mqe_t = col;
                        if (col == tl1) score16 = h;
                    }
                }
            }
            int mqe = mqe_t >= 0 ? mqe16 >> 4 : AW_NEG_INF;
            int mte = mte_q >= 0 ? mte16 >> 4 : AW_NEG_INF;
            int score = score16 != INT_MIN ? score16 >> 4 : AW_NEG_INF;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int ov = __shfl_xor_sync(FULLMASK, mqe, o), op = __shfl_xor_sync(FULLMASK, mqe_t, o);
                best_merge(mqe, mqe_t, ov, op);
                const int tv = __shfl_xor_sync(FULLMASK, mte, o), tp = __shfl_xor_sync(FULLMASK, mte_q, o);
                best_merge(mte, mte_q, tv, tp);
                score = max(score, __shfl_xor_sync(FULLMASK, score, o));
            }
            if (!last) {
                // the pair's record first, then the H that lets the right neighbour read it
                if (lane == 0) atomicMax(&A.res[idx].mqe_key, mqe_key(mqe, mqe_t));
                __threadfence();
                __syncwarp();
                if (C.bnd) bnd_store(C.bnd + qlen, (uint32_t)h, 0u);
            } else if (lane == 0) {
                if (nstrip > 1) {
                    const unsigned long long k = *(volatile unsigned long long *)&A.res[idx].mqe_key;
                    best_merge(mqe, mqe_t, (int)((uint32_t)(k >> 32) ^ 0x80000000u), (int)(uint32_t)k);
                }
                KswOut o;
                o.score = score, o.max = 0, o.max_q = -1, o.max_t = -1;
                o.mqe = mqe, o.mqe_t = mqe_t, o.mte = mte, o.mte_q = mte_q;
                o.n_cigar = 0, o.zdropped = 0, o.reach_end = 0, o.stopped = 0;
                A.out[idx] = o;
            }
        }
        if (failed) break;
    }
}

// ---- traceback -------------------------------------------------------------

template <int NP, bool TRK>
struct BtShape {
    static constexpr int CPW = NP == 8 ? 8 : 4, WB = CPW * (TRK ? 2 : 1);
    using Window = TbWindow<WB, CPW, TRK ? 1 : 0, true>;
    using Probe = TbWindow<WB, CPW, 0, false>;  // the rows and columns of a Singletrack gap search
    static constexpr int WARPS = TRK ? 1 : 4;
    static constexpr int BYTES = Window::BYTES + (TRK ? Probe::BYTES : 0);
};

struct FullBtArgs {
    const KswPair *pairs;
    const int32_t *order;
    int n, flag, m;
    const uint8_t *tb, *qcodes, *tcodes;
    KswOut *out;
    uint32_t *cig;
    KswScore sc;
    int8_t mat[64];
};

// ksw_backtrack of minimap2/ksw2.h:160-192 over the strip layout, or the Singletrack
// reconstruction; in full mode every visited cell is a stored cell, so the off/off_end forcing
// never fires.  One warp per pair walks in runs over prefetched tiles (tb_walk.cuh).
template <int NP, bool TRK>
__global__ void __launch_bounds__(32 * BtShape<NP, TRK>::WARPS) ksw_backtrack_full_kernel(FullBtArgs A) {
    using Sh = BtShape<NP, TRK>;
    __shared__ __align__(16) uint8_t tiles[Sh::WARPS][Sh::BYTES];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pi = blockIdx.x * Sh::WARPS + warp;
    if (pi >= A.n) return;
    const int idx = A.order[pi], flag = A.flag;
    const KswPair P = A.pairs[idx];
    KswOut o = A.out[idx];
    const int qlen = P.qlen, tlen = P.tlen;
    int i = tlen - 1, j = qlen - 1, state = 0;
    if (o.zdropped || o.stopped) return;
    if (!TRK && (flag & AW_EZ_SEMIGLOBAL_END)) {
        if (o.mqe > o.mte) o.score = o.mqe, i = o.mqe_t, j = qlen - 1;
        else o.score = o.mte, i = tlen - 1, j = o.mte_q;
    }
    const uint8_t *tb = A.tb + P.tb_off;
    const int64_t steps = qlen + KSW_LAG;
    // words per lane-step of the layout, and the step at which row 0 of a word is stored
    constexpr int WPL = 2 * NP / Sh::CPW;
    typename Sh::Window win;
    win.init(tiles[warp], 32 * WPL * Sh::WB);
    auto grp = [&](int gg) -> TbGroup {
        if (gg < 0 || gg * Sh::CPW >= tlen) return TbGroup{tb, 0, -1};
        const int s = gg / (32 * WPL), g = gg % (32 * WPL), k = WPL == 2 ? g : 2 * g + 1;
        return TbGroup{tb + (((int64_t)s * steps + k) * (32 * WPL) + g) * Sh::WB, 0, qlen - 1};
    };
    auto inside = [](int, int) { return -1; };
    auto no_fill = [](int, int) {};
    WarpCigar w{A.cig + P.cig_off, 0, 0, 0};
    if constexpr (TRK) {
        typename Sh::Probe probe;
        probe.init(tiles[warp] + Sh::Window::BYTES, 32 * WPL * Sh::WB);
        if (tb_singletrack(i, j, w, win, probe, grp, inside, no_fill, A.sc, A.mat, A.m, A.qcodes + P.qoff, A.tcodes + P.toff)) {
            if (i >= 0) w.push(2, i + 1);
            if (j >= 0) w.push(1, j + 1);
            o.n_cigar = w.finish(true);
        }
        if (o.n_cigar == 0) o.zdropped = 1;
    } else {
        tb_walk(i, j, state, 0, w, win, grp, inside, no_fill);
        if (i >= 0) w.push(2, i + 1);
        if (j >= 0) w.push(1, j + 1);
        o.n_cigar = w.finish(!(flag & AW_EZ_REV_CIGAR));
    }
    if (lane == 0) A.out[idx] = o;
}

// Copy each pair's CIGAR from its slot to a packed buffer (one warp per pair).
__global__ void ksw_pack_cigar_kernel(const KswPair *pairs, int n, const KswOut *out,
                                      const uint32_t *cig, const int64_t *packed_off,
                                      uint32_t *packed) {
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= n) return;
    const int nc = out[wid].n_cigar;
    const uint32_t *src = cig + pairs[wid].cig_off;
    uint32_t *dst = packed + packed_off[wid];
    for (int i = lane; i < nc; i += 32) dst[i] = src[i];
}

// The kernel of a call and its dynamic shared memory (the score profiles of a CTA's warps).
typedef void (*FullKernel)(KswFullArgs);
template <int NP>
FullKernel full_kernel_np(int flag) {
    if (flag & AW_EZ_SCORE_ONLY) return ksw_full_kernel<SCORES, NP>;
    if (flag & AW_EZ_SINGLETRACK) return ksw_full_kernel<TRACKS, NP>;
    return (flag & AW_EZ_RIGHT) ? ksw_full_kernel<RIGHTMOST, NP> : ksw_full_kernel<LEFT, NP>;
}
FullKernel full_kernel(int flag, bool narrow) { return narrow ? full_kernel_np<2>(flag) : full_kernel_np<8>(flag); }
int full_smem(bool narrow) { return narrow ? cta_warps<2>() * Prof<2>::WARP : cta_warps<8>() * Prof<8>::WARP; }

// The dynamic shared memory limit is an attribute of a kernel on a device: set once.
cudaError_t full_prepare(int flag, bool narrow) {
    static std::atomic<uint32_t> set_on[4];
    if (narrow) return cudaSuccess;  // below the default limit
    int dev = 0;
    cudaGetDevice(&dev);
    const int mode = (flag & AW_EZ_SCORE_ONLY) ? SCORES : (flag & AW_EZ_SINGLETRACK) ? TRACKS : (flag & AW_EZ_RIGHT) ? RIGHTMOST : LEFT;
    const uint32_t bit = 1u << (dev & 31);
    if (set_on[mode].load() & bit) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(full_kernel(flag, narrow), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               full_smem(narrow));
    if (e == cudaSuccess) set_on[mode].fetch_or(bit);
    return e;
}

template <int NP, bool TRK>
void launch_bt(const FullBtArgs &a, cudaStream_t st) {
    constexpr int W = BtShape<NP, TRK>::WARPS;
    ksw_backtrack_full_kernel<NP, TRK><<<(a.n + W - 1) / W, 32 * W, 0, st>>>(a);
}

}  // namespace

int ksw_full_warps_per_cta(bool narrow) { return narrow ? cta_warps<2>() : cta_warps<8>(); }

int ksw_full_occupancy(int flag, bool narrow) {
    // CTAs per SM depend only on the instantiation: cached per device
    static std::atomic<int> cache[16][4][2];
    int dev = 0;
    cudaGetDevice(&dev);
    const int mode = (flag & AW_EZ_SCORE_ONLY) ? SCORES : (flag & AW_EZ_SINGLETRACK) ? TRACKS : (flag & AW_EZ_RIGHT) ? RIGHTMOST : LEFT;
    std::atomic<int> *slot = dev >= 0 && dev < 16 ? &cache[dev][mode][narrow ? 1 : 0] : nullptr;
    if (slot && slot->load() > 0) return slot->load();
    int nb = 0;
    if (full_prepare(flag, narrow) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, full_kernel(flag, narrow), 32 * ksw_full_warps_per_cta(narrow),
                                                      full_smem(narrow)) != cudaSuccess)
        return 0;
    if (slot) slot->store(nb);
    return nb;
}

cudaError_t launch_ksw_full(const KswFullArgs &a, int flag, bool narrow, int ctas, cudaStream_t st) {
    if (a.n <= 0) return cudaSuccess;
    const cudaError_t e = full_prepare(flag, narrow);
    if (e != cudaSuccess) return e;
    full_kernel(flag, narrow)<<<ctas, 32 * ksw_full_warps_per_cta(narrow), full_smem(narrow), st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_ksw_backtrack_full(const KswPair *pairs, const int32_t *order, int n,
                                      const uint8_t *tb, KswOut *out, uint32_t *cig, int flag, bool narrow,
                                      const uint8_t *qcodes, const uint8_t *tcodes, const KswScore &S,
                                      const int8_t *mat, int m, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    FullBtArgs a;
    a.pairs = pairs, a.order = order, a.n = n, a.flag = flag, a.m = m;
    a.tb = tb, a.qcodes = qcodes, a.tcodes = tcodes, a.out = out, a.cig = cig, a.sc = S;
    memset(a.mat, 0, sizeof(a.mat));
    memcpy(a.mat, mat, (size_t)m * m);
    if (flag & AW_EZ_SINGLETRACK) narrow ? launch_bt<2, true>(a, st) : launch_bt<8, true>(a, st);
    else narrow ? launch_bt<2, false>(a, st) : launch_bt<8, false>(a, st);
    return cudaGetLastError();
}

__global__ void set_deadline_kernel(unsigned long long *d, unsigned long long remaining_ns) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    *d = remaining_ns == ~0ull ? ~0ull : t + remaining_ns;
}

cudaError_t launch_set_deadline(unsigned long long *deadline, unsigned long long remaining_ns, cudaStream_t st) {
    set_deadline_kernel<<<1, 1, 0, st>>>(deadline, remaining_ns);
    return cudaGetLastError();
}

cudaError_t launch_ksw_pack_cigar(const KswPair *pairs, int n, const KswOut *out,
                                  const uint32_t *cig, const int64_t *packed_off, uint32_t *packed,
                                  cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int threads = 256;
    const int blocks = (int)(((int64_t)n * 32 + threads - 1) / threads);
    ksw_pack_cigar_kernel<<<blocks, threads, 0, st>>>(pairs, n, out, cig, packed_off, packed);
    return cudaGetLastError();
}

}  // namespace aw
