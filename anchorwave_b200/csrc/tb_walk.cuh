// Warp-cooperative traceback reads for the strip layouts.
//
// A traceback walk (ksw_backtrack, the Singletrack reconstruction) is a chain of
// dependent decisions that moves up and left through the matrix.  Read one byte at a time
// it costs a shared-memory latency and a branch per cell (125 ns measured).  Here the 32
// lanes of a warp look at the next 32 cells of the walk's current direction at once: down
// the diagonal while the state is M, along the row or column inside a gap; a ballot gives
// the length of the run that the serial walk would take, so the walk advances a whole run
// per round and only changes of state are serial.
//
// The cells come from tiles of 32 rows x 64 columns in shared memory.  A walk mostly
// follows the diagonal, so while a tile is walked the next three down the diagonal are on
// their way (cp.async, one group per tile); each is placed 16 columns ahead of the
// diagonal, so that it still covers the walk after a drift of 16 columns either way.  A
// larger drift is a miss: the tile at the walk's position is fetched and the tiles ahead of
// it again.  Bound by the tiles' latency; measured against byte-by-byte walks over tiles
// fetched on a miss: one 5 kb pair 1.25 -> 0.14 ms, 768 pairs of 0.2-20 kb 6.8 -> 0.8 ms, four
// banded pairs of 60-160 kb 85 -> 10 ms, 128 Singletrack pairs of 2-8 kb 6.6 -> 0.6 ms.
#pragma once
#include <stdint.h>
#include <climits>
#include "aw_internal.h"

namespace aw {

// The stored rows of one column group: row jlo's word lies at p, the others `stride` (of the
// layout) apart; no row is stored when jhi < jlo.
struct TbGroup {
    const uint8_t *p;
    int jlo, jhi;
};

template <int WB>
__device__ __forceinline__ void tb_copy(uint32_t dst, const uint8_t *src, bool ok) {
    // zero bytes read (the word becomes zero) when the cell is not stored
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(WB), "r"(ok ? WB : 0)
                 : "memory");
}
__device__ __forceinline__ void tb_wait(int pending) {
    if (pending <= 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
    else if (pending == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else if (pending == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else asm volatile("cp.async.wait_group 3;" ::: "memory");
}

// WB: bytes per word (4, 8 or 16) covering CPW columns (Singletrack words hold the v bytes,
// then the u bytes); DEPTH: rows below a cell's own that a look at it needs as well.
// AHEAD: fetch the tiles down the diagonal ahead of the walk (four slots, else two).
template <int WB, int CPW, int DEPTH, bool AHEAD>
struct TbWindow {
    static constexpr int TR = 32, TG = 64 / CPW, PITCH = TR - DEPTH;
    static constexpr int RS = TG * WB + (WB == 16 ? 16 : 8);  // row stride: a diagonal spreads over the banks
    static constexpr int NS = AHEAD ? 4 : 2, SLOT = TR * RS, BYTES = NS * SLOT;
    const uint8_t *sm;
    uint32_t sa;
    int64_t stride;   // bytes between a group's rows in the layout
    int cur, cg, cj;  // the current tile: slot, last column group, last row
    int og, oj, oseq; // lane s < NS: the same of slot s, and its number
    int issued;       // tiles fetched so far (tile n lies in slot n % NS)

    __device__ void init(uint8_t *smem, int64_t row_stride) {
        sm = smem, sa = (uint32_t)__cvta_generic_to_shared(smem), stride = row_stride;
        reset();
    }
    // Forgets every tile (no copy may be under way).
    __device__ void reset() { cur = 0, cg = cj = INT_MIN / 2, og = oj = INT_MIN / 2, oseq = -1, issued = 0; }

    // Starts the copy of the tile whose last cell is (group g, row j); GRP(gg) describes group gg.
    template <class GRP>
    __device__ void fetch(int g, int j, GRP &&grp) {
        const int lane = threadIdx.x & 31, slot = issued % NS;
        if (j >= 0) {
            const TbGroup G = grp(g - lane % TG);
            constexpr int RPI = 32 / TG;
            const uint32_t dst = sa + slot * SLOT + (lane / TG) * RS + (lane % TG) * WB;
#pragma unroll 4
            for (int it = 0; it < TR / RPI; ++it) {
                const int row = j - (it * RPI + lane / TG);
                const bool ok = row >= G.jlo && row <= G.jhi;
                tb_copy<WB>(dst + it * RPI * RS, G.p + (ok ? (int64_t)(row - G.jlo) * stride : 0), ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (lane == slot) og = g, oj = j, oseq = issued;
        ++issued;
    }

    // Makes the tile that covers (i, j) and (i, j - DEPTH) the current one.
    template <class GRP>
    __device__ void ensure(int i, int j, GRP &&grp) {
        const int g = i / CPW, jd = max(j - DEPTH, 0);
        if (g <= cg && g > cg - TG && j <= cj && jd > cj - TR) return;
        const int lane = threadIdx.x & 31;
        __syncwarp();
        const unsigned b = __ballot_sync(0xffffffffu, lane < NS && g <= og && g > og - TG && j <= oj && jd > oj - TR);
        int seq;
        if (b) {
            cur = __ffs(b) - 1;
            seq = __shfl_sync(0xffffffffu, oseq, cur);
            cg = __shfl_sync(0xffffffffu, og, cur), cj = __shfl_sync(0xffffffffu, oj, cur);
        } else {
            tb_wait(0);  // a slot may only be refilled once its copy is done
            __syncwarp();
            seq = issued, cur = issued % NS, cg = g, cj = j;
            fetch(g, j, grp);
        }
        if (AHEAD) {
            // older tiles are complete with this one, so their slots are free again
            if (b) tb_wait(issued - 1 - seq), __syncwarp();
            while (issued - 1 - seq < NS - 1) {
                const int row = cj - PITCH * (issued - seq);
                fetch(max(i - (j - row) + 16, 0) / CPW, row, grp);
            }
            if (!b) tb_wait(issued - 1 - seq);
        } else {
            tb_wait(0);
        }
        __syncwarp();
    }

    // Makes the tile whose last cell is (i, j)'s group and row the current one.
    template <class GRP>
    __device__ void corner(int i, int j, GRP &&grp) {
        const int g = i / CPW;
        if (g == cg && j == cj) return;
        __syncwarp();
        const unsigned b = __ballot_sync(0xffffffffu, (threadIdx.x & 31) < NS && g == og && j == oj);
        cur = b ? __ffs(b) - 1 : issued % NS, cg = g, cj = j;
        if (!b) fetch(g, j, grp), tb_wait(0);
        __syncwarp();
    }

    // Whether (i, j) and (i, j - DEPTH) lie in the current tile (rows above the matrix count).
    __device__ __forceinline__ bool has(int i, int j) const {
        return i / CPW > cg - TG && max(j - DEPTH, 0) > cj - TR;
    }
    // Byte of the cell (i, j) of the current tile (part 1: the second half of the word).
    __device__ __forceinline__ uint32_t at(int i, int j, int part = 0) const {
        return sm[cur * SLOT + (cj - j) * RS + (cg - i / CPW) * WB + part * CPW + i % CPW];
    }
};

constexpr unsigned TB_ALL = 0xffffffffu;

// CIGAR under construction, replicated in every lane of the walking warp: the open
// run stays in registers and lane 0 writes a run when the next op differs (the
// merge rule of ksw_push_cigar, minimap2/ksw2.h:144-154).
struct WarpCigar {
    uint32_t *buf;
    int n;         // runs written
    uint32_t op;   // open run
    int len;       // 0 = no open run
    __device__ void push(uint32_t o, int l) {
        if (len > 0 && o == op) {
            len += l;
            return;
        }
        if (len > 0 && (threadIdx.x & 31) == 0) buf[n] = (uint32_t)len << 4 | op;
        if (len > 0) ++n;
        op = o, len = l;
    }
    __device__ int finish(bool reverse) {
        if (len > 0) {
            if ((threadIdx.x & 31) == 0) buf[n] = (uint32_t)len << 4 | op;
            ++n, len = 0;
        }
        __syncwarp();
        if (reverse) {
            const int lane = threadIdx.x & 31;
            for (int a = lane; a < n / 2; a += 32) {
                const uint32_t t = buf[a];
                buf[a] = buf[n - 1 - a], buf[n - 1 - a] = t;
            }
            __syncwarp();
        }
        return n;
    }
};

// ksw_backtrack (minimap2/ksw2.h:160-192) from (i, j) until the walk leaves the matrix or the
// columns >= col_lo, in runs.  FORCE(i, j): the move forced outside the computed band (1:
// deletion, 2: insertion), -1, or -2 for a cell whose bytes FILL(i, j) has to compute first.
template <class Window, class GRP, class FORCE, class FILL, class Cig>
__device__ void tb_walk(int &i, int &j, int &state, int col_lo, Cig &cg, Window &win, GRP &&grp, FORCE &&force,
                        FILL &&fill) {
    const int lane = threadIdx.x & 31;
    while (i >= 0 && j >= 0 && i >= col_lo) {
        win.ensure(i, j, grp);
        const int di = state == 0 || state == 1 || state == 3, dj = state == 0 || state == 2 || state == 4;
        const int li = i - (di ? lane : 0), lj = j - (dj ? lane : 0);
        const bool in = li >= 0 && lj >= 0 && li >= col_lo && win.has(li, lj);
        const int fc = in ? force(li, lj) : -1;
        const uint32_t c = in && fc == -1 ? win.at(li, lj) : 0u;
        // the cell takes the walk's state on: an M cell in state 0, a continued gap otherwise
        const bool on = in && fc == -1 && (state == 0 ? (c & 7u) == 0 : ((c >> (state + 2)) & 1u) != 0);
        const unsigned off = __ballot_sync(TB_ALL, !on);
        const int run = off ? __ffs(off) - 1 : 32;
        if (run > 0) {
            cg.push(state == 0 ? 0u : di ? 2u : 1u, run);
            i -= di ? run : 0, j -= dj ? run : 0;
        }
        // the cell that ends the run, if it is there: a forced move, or its own state
        if (run == 32 || !__shfl_sync(TB_ALL, in ? 1 : 0, run)) continue;
        const int f = __shfl_sync(TB_ALL, fc, run);
        if (f == -2) {
            if (run == 0) {
                tb_wait(0);
                fill(i, j);
                win.reset();
            }
            continue;
        }
        state = f >= 0 ? f : (int)(__shfl_sync(TB_ALL, c, run) & 7u);
        if (state == 0) continue;  // an M cell after a gap: the next round takes its run
        if (state == 1 || state == 3) cg.push(2, 1), --i;
        else cg.push(1, 1), --j;
    }
}

__device__ __forceinline__ int tb_sx8(uint32_t w) { return (int)(int8_t)(uint8_t)w; }
__device__ __forceinline__ int tb_st_gap(int l, int o1, int e1, int o2, int e2) {
    if (l <= 0) return 0;
    const long long a = (long long)o1 + (long long)l * e1, b = (long long)o2 + (long long)l * e2;
    return (int)(a > b ? a : b);
}

// The Singletrack reconstruction (minimap2/ksw2_singletrack.cpp:63-176) from (i, j) to a matrix
// edge.  FORCE as above (insertions above the computed blocks of an anti-diagonal, deletions
// below), FILL too.  Returns false when no gap explains a cell.  `probe` holds the tiles of a gap
// search.
template <class Window, class Probe, class GRP, class FORCE, class FILL>
__device__ bool tb_singletrack(int &i, int &j, WarpCigar &cg, Window &win, Probe &probe, GRP &&grp, FORCE &&force,
                               FILL &&fill, const KswScore &S, const int8_t *mat, int m, const uint8_t *qs, const uint8_t *ts) {
    const int lane = threadIdx.x & 31;
    auto stored = [&](int a, int b) { return force(a, b) < 0; };
    const int o1 = -S.q, g1 = -S.e, o2 = -S.q2, g2 = -S.e2;
    auto fill_at = [&](int a, int b) {
        tb_wait(0);
        fill(a, b);
        win.reset(), probe.reset();
    };
    // the difference along the matrix edge for edge cell c
    auto edge = [&](int c) { return tb_st_gap(c + 1, o1, g1, o2, g2) - tb_st_gap(c, o1, g1, o2, g2); };
    while (i >= 0 && j >= 0) {
        const int f = force(i, j);
        if (f == 2) { cg.push(1, 1); --j; continue; }
        if (f == 1) { cg.push(2, 1); --i; continue; }
        if (f == -2 || (j > 0 && force(i, j - 1) == -2)) {
            fill_at(i, f == -2 ? j : j - 1);
            continue;
        }
        // the run of diagonal moves: v(i, j) + u(i, j-1) is the cell's substitution score
        win.ensure(i, j, grp);
        const int li = i - lane, lj = j - lane;
        const bool in = li >= 0 && lj >= 0 && win.has(li, lj) && stored(li, lj) &&
                        force(li, lj) != -2 && (lj == 0 || force(li, lj - 1) != -2);
        bool on = in;
        if (in) {
            const int h = tb_sx8(win.at(li, lj, 0));
            const bool fin = lj == 0 || stored(li, lj - 1);
            const int v = lj == 0 ? edge(li) : fin ? tb_sx8(win.at(li, lj - 1, 1)) : 0;
            on = fin && h + v == mat[ts[li] * m + qs[lj]];
        }
        const unsigned off = __ballot_sync(TB_ALL, !on);
        const int run = off ? __ffs(off) - 1 : 32;
        if (run > 0) {
            cg.push(0, run);
            i -= run, j -= run;
        }
        if (run == 32 || !__shfl_sync(TB_ALL, in ? 1 : 0, run)) continue;
        // the gap that leaves (i, j): the first length l whose summed differences up the
        // column of rows (insertion) or along the row (deletion) are exactly a gap of l;
        // 32 lengths at a time, lane k looking at length base + k + 1.  Sums over cells
        // outside the stored band match no gap (d_ok, i_ok).
        int base = 0, dsum = 0, isum = 0;
        bool d_ok = true, i_ok = true;
        for (;;) {
            const int l = base + lane + 1, id = i - l, jn = j - l;
            // lengths from the first cell on that is not computed yet do not count (the cells above
            // (i, j) were computed with it)
            const unsigned nb = __ballot_sync(TB_ALL, d_ok && id + 1 >= 0 && force(id + 1, j) == -2);
            const unsigned known = nb ? (nb & (0u - nb)) - 1u : TB_ALL;
            // differences of the l-th cell: u(i-l+1, j) and v(i, j-l+1)
            int du = 0, dv = 0;
            bool uf = true, vf = true;
            if (d_ok && i - base >= 0) probe.corner(i - base, j, grp);
            if (d_ok && id + 1 >= 0) {
                uf = stored(id + 1, j);
                if (uf) du = tb_sx8(probe.at(id + 1, j, 1));
            }
            __syncwarp();
            if (i_ok && j - base >= 0) probe.corner(i, j - base, grp);
            if (i_ok && jn + 1 >= 0) {
                vf = stored(i, jn + 1);
                if (vf) dv = tb_sx8(probe.at(i, jn + 1, 0));
            }
            __syncwarp();
#pragma unroll
            for (int k = 1; k < 32; k <<= 1) {
                const int a = __shfl_up_sync(TB_ALL, du, k), b = __shfl_up_sync(TB_ALL, dv, k);
                if (lane >= k) du += a, dv += b;
            }
            const unsigned ub = __ballot_sync(TB_ALL, !uf), vb = __ballot_sync(TB_ALL, !vf);
            const unsigned upto = lane == 31 ? TB_ALL : (2u << lane) - 1u;
            const int a1 = o1 + l * g1, a2 = o2 + l * g2, dd = dsum + du, di = isum + dv;
            const bool dhit = d_ok && !(ub & upto) && id >= -1 && (dd == a1 || dd == a2);
            const bool ihit = i_ok && !(vb & upto) && jn >= -1 && (di == a1 || di == a2);
            const unsigned end = __ballot_sync(TB_ALL, l > i + 1 && l > j + 1) & known;
            const unsigned db = __ballot_sync(TB_ALL, dhit), hit = (db | __ballot_sync(TB_ALL, ihit)) & known;
            if (hit && (!end || __ffs(hit) <= __ffs(end))) {
                const int k = __ffs(hit) - 1, len = base + k + 1;
                if (db >> k & 1u) cg.push(2, len), i -= len;
                else cg.push(1, len), j -= len;
                break;
            }
            if (end) return false;
            if (nb) {
                fill_at(i - base - (__ffs(nb) - 1), j);
                continue;
            }
            dsum += __shfl_sync(TB_ALL, du, 31), isum += __shfl_sync(TB_ALL, dv, 31);
            d_ok = d_ok && !ub, i_ok = i_ok && !vb;
            base += 32;
        }
    }
    return true;
}

}  // namespace aw
