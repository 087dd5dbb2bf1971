// The KSW2 extd2 cell on two 16-bit fields per register, shared by the full-matrix and the
// banded strip kernels (minimap2/ksw2_extd2_sse.c:43-71 + :237-330).
#pragma once
#include "aw_internal.h"

namespace aw {

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// Difference along a matrix edge for edge cell index r (ksw2_extd2_sse.c:167,171).
__device__ __forceinline__ int edge_diff(int r, const KswScore &S) {
    return r == 0 ? -S.qe : r < S.long_thres ? -S.e : r == S.long_thres ? S.long_diff : -S.e2;
}

// ---- packed cell fields ------------------------------------------------------------
// Every field holds 16*value + FB; x, y, x2, y2 carry their candidate's priority tag on
// top (so x + v is already the tagged candidate a), and the score carries 2*FB + its tag.
// Every 32-bit add below keeps each field inside [0, 65536), and every value a DPX op compares
// inside [0, 32768), while no candidate is above CAND_MAX.  The other bounds hold for any cell,
// also the ones outside a band that have no consistent neighbours, whatever x and y are: with
// u, v in [-M, mch + M] before a step (M = q + e, or the largest difference along a matrix edge,
// -long_diff, where e = e2; the initial and the boundary values are, and mch < 0 moves the bounds
// by -mch at most), z = min(max(s, a, ...), mch) is either mch, and then z - v >= -M, or at least
// a = x + v >= v - (q + e), and then z - v >= -(q + e); z - v <= mch + M since v >= -M; the same for
// z - u.  x, y >= -(q + e) and x2, y2 >= -(q2 + e2) by their max, M <= q2 + e2 and mch <= 0.  So by
// the magnitude bound of full_path_ok (both gaps, the mismatch and the match together at most 100)
// no field falls below -256 * 16.
// In a full matrix x <= q and so on; at the edge of a band they may grow by M - e a step (max(a - z -
// e, ..) with a = x + v, where z is clipped to mch), which the banded kernel checks.
// The adds are 2-input multiply-adds by a runtime one (or minus one), so they issue on the
// FMA pipe and leave the ALU pipe to the max/min/permute work.
constexpr int FB = 4096;  // a multiple of 16 * 256: the byte above a field's tag is the value
constexpr int CAND_MAX = (32768 - 2 * FB) / 16 - 1;
// A constant in both fields: for 32-bit adds (c * 65537, so that a negative c borrows
// exactly what the field sum carries back) and for SIMD operands (each field = c).
__host__ __device__ constexpr uint32_t add2(int c) { return (uint32_t)c * 0x10001u; }
__host__ __device__ constexpr uint32_t rep2(int c) { return ((uint32_t)c & 0xffffu) * 0x10001u; }

// What a sweep keeps for the traceback: nothing, the state bytes under the left-aligned or the
// right-aligned tie rule, or the Singletrack tracks.
enum { SCORES = 0, LEFT = 1, RIGHTMOST = 2, TRACKS = 3 };

// Priority tags of the candidates s, a, b, a2, b2 (the larger tag wins a tie of values),
// and the XOR that turns the winning tag into the reference's state code d (0 = s, 1 = a,
// 2 = b, 3 = a2, 4 = b2).  Score-only sweeps need no arg-max: no tags.
template <int MODE>
struct Tags {
    static constexpr bool CIGAR = MODE == LEFT || MODE == RIGHTMOST, RIGHT = MODE == RIGHTMOST;
    static constexpr int s = !CIGAR ? 0 : RIGHT ? 0 : 7;
    static constexpr int a = !CIGAR ? 0 : RIGHT ? 1 : 6;
    static constexpr int b = !CIGAR ? 0 : RIGHT ? 2 : 5;
    static constexpr int a2 = !CIGAR ? 0 : RIGHT ? 3 : 4;
    static constexpr int b2 = !CIGAR ? 0 : RIGHT ? 4 : 3;
    static constexpr uint32_t dx = (CIGAR && !RIGHT) ? 0x00070007u : 0u;
};

// Per-launch packed constants of the cell.
struct CellK {
    uint32_t ke, ke2;               // Ze = Z + ke: W = candidate - Ze = 16 (cand - z - e) + FB + tag
    uint32_t kxa, kxb, kxa2, kxb2;  // x' = max(W, kx): the field of -(q+e) (-(q2+e2)) with the tag (SIMD)
    uint32_t ca, cb, ca2, cb2;      // continuation: relu(min(W + c, 8 or 16))       (SIMD)
    uint32_t mch;                   // z = min(z, mch)                                (SIMD)
    uint32_t one, neg1;             // runtime 1 and -1 of the multiply-adds
};

template <int MODE>
__device__ __forceinline__ CellK make_cellk(const KswScore &S, uint32_t one) {
    using T = Tags<MODE>;
    constexpr bool RIGHT = T::RIGHT;
    CellK K;
    K.ke = add2(16 * S.e - FB), K.ke2 = add2(16 * S.e2 - FB);
    const int xa = FB - 16 * S.qe + T::a, xb = FB - 16 * S.qe + T::b;
    const int xa2 = FB - 16 * S.qe2 + T::a2, xb2 = FB - 16 * S.qe2 + T::b2;
    K.kxa = rep2(xa), K.kxb = rep2(xb), K.kxa2 = rep2(xa2), K.kxb2 = rep2(xb2);
    // left-aligned: a - z + q > 0 (ksw2_extd2_sse.c:268-271) <=> W - kx >= 16;
    // right-aligned: >= 0 (:315-318) <=> W - kx >= 0.  The a bit is 8, the others 16
    // (scaled to 32 and 64 when they are added to the state byte).
    K.ca = rep2((RIGHT ? 8 : -8) - xa), K.cb = rep2((RIGHT ? 16 : 0) - xb);
    K.ca2 = rep2((RIGHT ? 16 : 0) - xa2), K.cb2 = rep2((RIGHT ? 16 : 0) - xb2);
    K.mch = rep2(16 * S.mch + 2 * FB);
    K.one = one, K.neg1 = 0u - one;
    return K;
}

// Two cells, one per field.  In: sc (tagged score), X/V/X2 from the left column, U/Y/Y2
// the column state from the row above.  Out: X/V/X2 for the next column, U/Y/Y2 for
// the next row, D the two state bytes (one per field).  CHAIN: a warp alone, where the
// dependent steps count and not the balance of the pipes: 3-input adds instead of two
// multiply-adds each.
template <int MODE, bool CHAIN>
__device__ __forceinline__ void cell2(uint32_t sc, uint32_t &X, uint32_t &V, uint32_t &X2, uint32_t &U,
                                      uint32_t &Y, uint32_t &Y2, uint32_t &D, const CellK &K) {
    constexpr bool CIGAR = Tags<MODE>::CIGAR;
    // a = x + v, b = y + u, a2 = x2 + v, b2 = y2 + u (ksw2_extd2_sse.c:240-243), tagged
    const uint32_t A = CHAIN ? X + V : X * K.one + V, Bv = CHAIN ? Y + U : Y * K.one + U;
    const uint32_t A2 = CHAIN ? X2 + V : X2 * K.one + V, B2 = CHAIN ? Y2 + U : Y2 * K.one + U;
    uint32_t Z = __vimax3_s16x2(__vimax3_s16x2(sc, Bv, B2), A, A2);
    if (CIGAR) {
        D = (Z & 0x000f000fu) ^ Tags<MODE>::dx;
        Z &= 0xfff0fff0u;
    }
    Z = __vmins2(Z, K.mch);  // ksw2_extd2_sse.c:252
    const uint32_t Un = CHAIN ? Z - V : V * K.neg1 + Z, Vn = CHAIN ? Z - U : U * K.neg1 + Z;
    uint32_t Wa, Wb, Wa2, Wb2;
    if (CHAIN) {
        Wa = A - Z - K.ke, Wb = Bv - Z - K.ke, Wa2 = A2 - Z - K.ke2, Wb2 = B2 - Z - K.ke2;
    } else {
        const uint32_t Ze = Z * K.one + K.ke, Ze2 = Z * K.one + K.ke2;
        Wa = Ze * K.neg1 + A, Wb = Ze * K.neg1 + Bv, Wa2 = Ze2 * K.neg1 + A2, Wb2 = Ze2 * K.neg1 + B2;
    }
    X = __vmaxs2(Wa, K.kxa);
    Y = __vmaxs2(Wb, K.kxb);
    X2 = __vmaxs2(Wa2, K.kxa2);
    Y2 = __vmaxs2(Wb2, K.kxb2);
    if (CIGAR) {
        D = __viaddmin_s16x2_relu(Wa, K.ca, 0x00080008u) * K.one + D;
        D = __viaddmin_s16x2_relu(Wb, K.cb, 0x00100010u) * K.one + D;
        D = __viaddmin_s16x2_relu(Wa2, K.ca2, 0x00100010u) * 2u + D;
        D = __viaddmin_s16x2_relu(Wb2, K.cb2, 0x00100010u) * 4u + D;
    }
    U = Un;
    V = Vn;
}

__device__ __forceinline__ int fld(uint32_t w, int f) { return f ? (int)(w >> 16) : (int)(w & 0xffffu); }


}  // namespace aw
