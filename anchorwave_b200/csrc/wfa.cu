// Gap-affine-2p end-to-end WFA (WFA2-lib as AnchorWave configures it:
// src/myImportandFunction/WfaAlignment.cpp:143-170) on sm_100a.
//
// A warp, a CTA or a cluster of CTAs per pair, by length; its threads cover the diagonals of a
// wavefront.  Per score s:
//   * extend M[s] (wavefront/wavefront_extend.c:86-121): each lane advances its
//     diagonal by comparing 16, then 32 bases of pattern and text at a time in 2-bit copies
//     of the sequences (the run also ends at the end of either sequence); pairs with any byte
//     other than A, C, G, T (the reference compares raw characters) compare 8 bytes at a time
//     instead, where the sentinels after each sequence ('!' pattern, '?' text,
//     wavefront/wavefront_sequences.c:37-39) stop the run;
//   * end-to-end check on diagonal tlen-plen (wavefront/wavefront_termination.c:37-60);
//   * compute s+1 from M[s-x], M[s-o1-e1], I1/D1[s-e1], M[s-o2-e2], I2/D2[s-e2]
//     (wavefront/wavefront_compute_affine2p.c:45-106) over the limits of
//     wavefront/wavefront_compute.c:56-105 (a missing input counts as the null
//     wavefront lo=1, hi=-1), allocating I/D outputs only when one of their
//     inputs exists (:459-572), then trimming out-of-matrix ends (:654-690).
// Values outside a wavefront's trimmed [lo, hi] read as NULL, which is what the
// reference's NULL end padding gives.  Standard mode retains every component of
// every score for the piggyback backtrace (wavefront/wavefront_backtrace.c:321-530);
// Singletrack keeps only M and recycles I/D through a ring of max(e1,e2)+1 slots,
// then reconstructs the path from M (:587-762).
// Medium and low memory (the piggyback modes, wavefront/wavefront_compute_affine2p.c:110-282)
// keep only the scores the compute step still reads (M: the last max_score_scope; I1/D1:
// the last e1+1; I2/D2: the last e2+1) in rings of slots; every cell carries the
// packed CIGAR of its latest operations and a link to the block that holds the earlier
// ones, and a cell whose packed CIGAR reaches 15 operations moves it into a new block
// (wavefront/wavefront_backtrace_offload.c); the traceback follows the links from the end
// cell and unpacks the blocks oldest first, re-extending the matches
// (wavefront/wavefront_backtrace.c:767-799, wavefront/wavefront_pcigar.c:222-278).
//
// Memory: per-score headers and wavefront arrays come from one device pool in 256 KiB
// chunks (larger arrays in several), taken from its end by an atomicAdd.  A finished pair
// gives its chunks to a free ring, from which the next pairs take theirs first, so a
// batch whose arrays fit a chunk needs the memory of the pairs in flight and not of all pairs
// (16,384 pairs of 0.1-10 kb in a 20 GB pool: 672 -> 123 ms, 33 rounds -> 1).  Larger arrays (the
// Singletrack I/D ring from 5.4 kb in sum, the piggyback rings from about 600 diagonals) always
// come from the end, and what one gives back serves as single chunks.  A pair that finds
// the pool empty stops with WFA_RETRY and the host re-runs it in a later round with a
// fresh pool, a pair alone in the least memory (WfaArgs::free_slots).
#include "aw_internal.h"
#include "wfa_internal.h"

#include <cooperative_groups.h>

namespace aw {
namespace {

constexpr int32_t WF_NULL = INT32_MIN / 2;
constexpr int HDR_CHUNK = 256;               // scores per header chunk

struct CompHdr {
    int32_t lo, hi, base, pad;
    int64_t off;  // byte offset of offsets[base] in the pool
};
struct ScoreHdr {
    CompHdr c[5];  // M, I1, D1, I2, D2
};
enum { CM = 0, CI1 = 1, CD1 = 2, CI2 = 3, CD2 = 4 };

// A pair's (or, for piggyback blocks, a warp's) memory: the current chunk's free range and the
// chunks taken, linked through their first 16 bytes (previous chunk, size).  In shared memory:
// one lane of a warp uses it, and every lane would pay for its registers.
struct Alloc {
    int64_t cur, end;
    int64_t from;   // the current chunk's first byte
    int64_t used;   // bytes allocated in the chunks before it
    int64_t list;
    __device__ void init() { cur = end = from = used = 0, list = -1; }
    // Bytes allocated: what a pair holds, whatever the chunks that they lie in.
    __device__ int64_t total() const { return used + (cur - from); }
};

// Packed CIGAR of the piggyback modes (wavefront/wavefront_pcigar.h:44-71): 2 bits per
// operation, newest lowest (1 deletion, 2 mismatch or gap close, 3 insertion).
constexpr uint32_t PC_ALMOST_FULL = 0x10000000u;  // 15 operations or more
constexpr uint32_t BT_NULL = 0xFFFFFFFFu;          // no earlier block
constexpr int PIG_U = 2;                           // diagonals per lane in flight
constexpr uint32_t LANE_BLOCKS = 32;               // blocks a lane reserves at a time
constexpr int64_t TIGHT_PIECE = 64 << 10;          // bytes taken at a time by a pair alone (WfaArgs::free_slots)

// The pool as the allocating functions (out of line, so no reference to the kernel's arguments)
// take it.
struct Pool {
    uint8_t *base;
    int64_t bytes;
    WfaPoolCtl *ctl;
    int32_t *ring;
    uint32_t slots;
};
__device__ __forceinline__ Pool pool_of(const WfaArgs &A) {
    return Pool{A.pool, A.pool_bytes, A.ctl, A.free_ring, A.free_slots};
}

__device__ __forceinline__ int64_t pool_grab(const Pool &A, int64_t bytes) {
    const unsigned long long b = atomicAdd(&A.ctl->head, (unsigned long long)bytes);
    if ((int64_t)(b + bytes) > A.bytes) return -1;
    return (int64_t)b;
}

// The same, but `bytes` becomes what is left of the pool if that is less, down to `least`.
__device__ __noinline__ int64_t pool_grab_rest(Pool A, int64_t &bytes, int64_t least) {
    for (int i = 0; i < 64; ++i) {
        const int64_t h = *(volatile int64_t *)&A.ctl->head;
        const int64_t len = min(bytes, (A.bytes - h) & ~(int64_t)255);
        if (len < least) return -1;
        if (atomicCAS(&A.ctl->head, (unsigned long long)h, (unsigned long long)(h + len)) != (unsigned long long)h) continue;
        bytes = len;
        return h;
    }
    return pool_grab(A, bytes);
}

// A chunk of a finished pair, or -1.  The ring holds `avail` complete entries; the entry at the
// taken position may still be on its way from the thread that reserved it, hence the wait.
__device__ __forceinline__ int64_t free_pop(const Pool &A) {
    if (*(volatile int32_t *)&A.ctl->avail <= 0) return -1;
    if (atomicSub(&A.ctl->avail, 1) <= 0) {
        atomicAdd(&A.ctl->avail, 1);
        return -1;
    }
    int32_t *slot = A.ring + atomicAdd(&A.ctl->popped, 1u) % A.slots;
    int32_t v = 0;
    for (int spins = 0; spins < (1 << 20) && (v = atomicExch(slot, 0)) == 0; ++spins) __nanosleep(20);
    __threadfence();  // the previous owner's accesses come before ours
    return v ? (int64_t)(v - 1) * WFA_CHUNK : -1;
}
__device__ __forceinline__ void free_push(const Pool &A, int64_t off) {
    int32_t *slot = A.ring + atomicAdd(&A.ctl->pushed, 1u) % A.slots;
    for (int spins = 0; atomicCAS(slot, 0, (int32_t)(off / WFA_CHUNK) + 1) != 0; ++spins) {
        if (spins > (1 << 20)) return;  // never with a slot per chunk; the chunk is lost for the round
        __nanosleep(20);
    }
    __threadfence();
    atomicAdd(&A.ctl->avail, 1);
}

// One thread: a chunk that holds `bytes`, linked to the allocation's list; false if there is none.
__device__ __noinline__ bool take_chunk(Pool A, Alloc &al, int64_t bytes) {
    if (A.slots == 0) {  // a pair alone
        const int64_t len = *(volatile int64_t *)&A.ctl->head + TIGHT_PIECE <= A.bytes ? max(bytes, TIGHT_PIECE) : bytes;
        const int64_t b = pool_grab(A, len);
        if (b < 0) return false;
        if (b == al.end) {  // the current piece grows
            al.end += len;
            return true;
        }
        al.used = al.total();
        al.cur = al.from = b, al.end = b + len;
        return true;
    }
    const int64_t sz = (bytes + 16 + WFA_CHUNK - 1) / WFA_CHUNK * WFA_CHUNK;
    int64_t b = sz == WFA_CHUNK ? free_pop(A) : -1;
    if (b < 0) b = pool_grab(A, sz);
    if (b < 0 && sz == WFA_CHUNK) b = free_pop(A);  // given back meanwhile
    if (b < 0) return false;
    int64_t *h = (int64_t *)(A.base + b);
    h[0] = al.list, h[1] = sz;
    al.used = al.total();
    al.list = b, al.cur = al.from = b + 16, al.end = b + sz;
    return true;
}

// One thread, after every access to the allocation: its chunks back to the pool.
__device__ __noinline__ void give_back(Pool A, Alloc &al) {
    __threadfence();
    for (int64_t b = al.list; b >= 0;) {
        const int64_t *h = (const int64_t *)(A.base + b);
        const int64_t prev = h[0], sz = h[1];
        for (int64_t o = 0; o < sz; o += WFA_CHUNK) free_push(A, b + o);
        b = prev;
    }
    al.list = -1;
}

// Lane-0 bump allocation inside the current chunk; broadcast to the warp (-1: none left).
__device__ __forceinline__ int64_t warp_alloc(const WfaArgs &A, Alloc &al, int64_t bytes, int lane) {
    bytes = (bytes + 15) & ~(int64_t)15;
    int64_t r = -1;
    if (lane == 0 && (al.cur + bytes <= al.end || take_chunk(pool_of(A), al, bytes))) {
        r = al.cur;
        al.cur = r + bytes;
    }
    return __shfl_sync(0xffffffffu, r, 0);
}

__device__ __forceinline__ ScoreHdr *hdr_ptr(const WfaArgs &A, const int64_t *ctab, int s) {
    return (ScoreHdr *)(A.pool + ctab[s / HDR_CHUNK]) + (s % HDR_CHUNK);
}

// The forward pass reads M's headers of the last max_score_scope scores, I1/D1's of the last
// e1 and I2/D2's of the last e2; each warp (or CTA) keeps them in shared-memory rings (powers
// of two, masks mm, m1, m2) as well as in the pool (the backtrace reads all of them from the
// pool).  mm < 0: pool only.
struct RingShape {
    int mm, m1, m2;
    __host__ __device__ int entries() const { return mm < 0 ? 0 : mm + 1 + 2 * (m1 + 1) + 2 * (m2 + 1); }
};
struct HdrRing {
    CompHdr *ring;
    RingShape sh;
    __device__ __forceinline__ CompHdr *at(int c, int sc) const {
        if (c == CM) return ring + (sc & sh.mm);
        CompHdr *r = ring + sh.mm + 1;
        if (c <= CD1) return r + (c - CI1) * (sh.m1 + 1) + (sc & sh.m1);
        return r + 2 * (sh.m1 + 1) + (c - CI2) * (sh.m2 + 1) + (sc & sh.m2);
    }
    __device__ __forceinline__ CompHdr get(const WfaArgs &A, const int64_t *ctab, int c, int sc) const {
        return sh.mm >= 0 ? *at(c, sc) : hdr_ptr(A, ctab, sc)->c[c];
    }
    __device__ __forceinline__ void put(int c, int sc, const CompHdr &h) const {
        if (sh.mm >= 0) *at(c, sc) = h;
    }
    __device__ __forceinline__ int mask(int c) const { return c == CM ? sh.mm : c <= CD1 ? sh.m1 : sh.m2; }
};

__device__ __forceinline__ int32_t getv(const WfaArgs &A, const CompHdr &h, int k) {
    if (k < h.lo || k > h.hi) return WF_NULL;
    return ((const int32_t *)(A.pool + h.off))[k - h.base];
}

// An input wavefront of the compute step: its range and the address of its diagonal 0 (the
// header's base folded in), so that a lane holds four values per input instead of six.
struct InHdr {
    int lo, hi;
    const int32_t *p;
};
__device__ __forceinline__ InHdr in_hdr(const WfaArgs &A, const CompHdr &h) {
    return InHdr{h.lo, h.hi, (const int32_t *)(A.pool + h.off) - h.base};
}
// As a predicated load, so that a lane's loads from several inputs are in flight together (the
// compiler made a branch of each check).
__device__ __forceinline__ int32_t getv(const InHdr &h, int k) {
    int32_t r;
    const int ok = k >= h.lo && k <= h.hi;
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; mov.b32 %0, %3; @q ld.global.b32 %0, [%1]; }"
                 : "=r"(r)
                 : "l"(h.p + k), "r"(ok), "n"(WF_NULL));
    return r;
}

// A piggyback cell: offset, packed CIGAR, link.  In a ring slot the three arrays of a
// component lie h.pad elements apart.
struct Cell {
    int32_t o;
    uint32_t pc, pv;
};
__device__ __forceinline__ Cell getc(const WfaArgs &A, const CompHdr &h, int k) {
    // three predicated loads: branches would put the cells of a lane one after the other
    Cell c;
    const int ok = k >= h.lo && k <= h.hi;
    const int32_t *p = (const int32_t *)(A.pool + h.off) + (k - h.base);
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %6, 0; mov.b32 %0, %7; mov.b32 %1, 0; mov.b32 %2, %8;"
                 " @q ld.global.b32 %0, [%3]; @q ld.global.b32 %1, [%4]; @q ld.global.b32 %2, [%5]; }"
                 : "=r"(c.o), "=r"(c.pc), "=r"(c.pv)
                 : "l"(p), "l"(p + h.pad), "l"(p + 2 * h.pad), "r"(ok), "n"(WF_NULL), "n"(BT_NULL));
    return c;
}

__device__ __forceinline__ uint64_t load8(const uint8_t *base, int64_t pos) {
    const uintptr_t a = (uintptr_t)(base + pos);
    const uint64_t *p = (const uint64_t *)(a & ~(uintptr_t)7);
    const int sh = (int)(a & 7) * 8;
    const uint64_t lo = p[0];
    if (!sh) return lo;
    return (lo >> sh) | (p[1] << (64 - sh));
}

// 32 bases from base g of a 2-bit arena (base i at bits 2*(i%32) of word i/32); the arena
// ends with a spare word.  SH: the words lie in shared memory.
template <bool SH = false>
__device__ __forceinline__ uint64_t load32b(const uint64_t *p, int g) {
    const int w = g >> 5, sh = (g & 31) * 2;
    const uint64_t lo = SH ? p[w] : __ldg(p + w), hi = SH ? p[w + 1] : __ldg(p + w + 1);
    return (lo >> sh) | ((hi << 1) << (63 - sh));
}
// 16 bases from base g, read as 32-bit words.
template <bool SH>
__device__ __forceinline__ uint32_t load16b(const uint32_t *p, int g) {
    const int w = g >> 4;
    return __funnelshift_r(SH ? p[w] : __ldg(p + w), SH ? p[w + 1] : __ldg(p + w + 1), 2 * g);
}
// A pair's sequences at 2 bits a base: the words that hold their first bases, and the places
// of those bases in them.
struct Bases {
    const uint64_t *p, *t;
    int po, to;
};
__device__ __forceinline__ Bases bases_of(const WfaArgs &A, const WfaPairDev &PR) {
    return Bases{A.ppat + (PR.poff >> 5), A.ptxt + (PR.toff >> 5), (int)(PR.poff & 31), (int)(PR.toff & 31)};
}

__device__ __forceinline__ bool in_matrix(int32_t o, int k, int plen, int tlen) {
    return (uint32_t)o <= (uint32_t)tlen && (uint32_t)(o - k) <= (uint32_t)plen;
}

// Length of the run of equal bases from pattern[v] / text[h], by the extend step's rules
// (2-bit words for ACGT-only pairs, else 8 bytes at a time up to the sentinels).
__device__ int64_t lcp1(const WfaArgs &A, const WfaPairDev &PR, const uint8_t *pat, const uint8_t *txt, int64_t v,
                        int64_t h) {
    const int64_t rem = min((int64_t)PR.plen - v, (int64_t)PR.tlen - h);
    if (rem <= 0) return 0;
    int64_t n = 0;
    if (PR.packed) {
        const Bases B = bases_of(A, PR);
        for (;;) {
            const uint64_t x = load32b(B.p, B.po + (int)(v + n)) ^ load32b(B.t, B.to + (int)(h + n));
            n += x ? (int64_t)((__ffsll((long long)x) - 1) >> 1) : 32;
            if (x || n >= rem) return min(n, rem);
        }
    }
    for (;;) {
        const uint64_t x = load8(pat, v + n) ^ load8(txt, h + n);
        if (x) return n + ((__ffsll((long long)x) - 1) >> 3);
        n += 8;
    }
}

__device__ __forceinline__ int64_t pb(int32_t o, int t) {
    return (int64_t)((((uint64_t)(int64_t)o) << 4) | (uint64_t)t);
}

struct OpsWriter {
    char *buf;
    int n, cap;
    bool ok;
    __device__ void put(char c, int times) {
        for (int i = 0; i < times; ++i) {
            if (n >= cap) { ok = false; return; }
            buf[n++] = c;
        }
    }
};

// Extends N diagonals of one lane at once (wavefront/wavefront_extend.c:86-121): o[u] is the
// offset on diagonal k0 + stride*u (WF_NULL: nothing to extend) and becomes the offset after the run
// of equal bases.  2-bit words (32 bases per XOR) for ACGT-only pairs; otherwise 8 bytes per
// XOR up to the sentinels after each sequence.  The N loads of a round are in flight together.
template <int N>
__device__ __forceinline__ bool any_of(const bool (&r)[N]) {
    bool a = false;
#pragma unroll
    for (int u = 0; u < N; ++u) a |= r[u];
    return a;
}

template <int N, bool SH = false>
__device__ __forceinline__ void extend_n(const WfaPairDev &PR, const Bases &B, const uint8_t *pat, const uint8_t *txt,
                                         int k0, int stride, int32_t (&o)[N]) {
    // o[u] is the text position h; the pattern position is h - k
    const int plen = PR.plen, tlen = PR.tlen;
    bool run[N];
#pragma unroll
    for (int u = 0; u < N; ++u) run[u] = o[u] != WF_NULL;
    if (PR.packed) {
        // the run ends at the first differing base or at the end of either sequence (the
        // sentinels of the byte path).  The first round compares 16 bases, in 32-bit words: most
        // runs are shorter; the others compare 32
        int rem[N];
        const uint32_t *wp = (const uint32_t *)B.p, *wt = (const uint32_t *)B.t;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            rem[u] = min(plen + (k0 + stride * u), tlen) - o[u];
            run[u] = run[u] && rem[u] > 0;
            uint32_t x = 1;
            if (run[u])
                x = load16b<SH>(wp, B.po + (o[u] - (k0 + stride * u))) ^ load16b<SH>(wt, B.to + o[u]);
            const int nb = run[u] ? min(__clz((int)__brev(x)) >> 1, rem[u]) : 0;
            o[u] += nb, rem[u] -= nb;
            run[u] = nb == 16 && rem[u] > 0;
        }
        while (any_of(run)) {
            uint64_t x[N];
#pragma unroll
            for (int u = 0; u < N; ++u)
                x[u] = run[u] ? load32b<SH>(B.p, B.po + (o[u] - (k0 + stride * u))) ^ load32b<SH>(B.t, B.to + o[u]) : 1;
#pragma unroll
            for (int u = 0; u < N; ++u) {
                const int nb = run[u] ? min(__clzll((long long)__brevll(x[u])) >> 1, rem[u]) : 0;
                o[u] += nb, rem[u] -= nb;
                run[u] = nb == 32 && rem[u] > 0;
            }
        }
        return;
    }
    bool any = any_of(run);
    while (any) {
        uint64_t x[N];
#pragma unroll
        for (int u = 0; u < N; ++u) x[u] = run[u] ? (load8(pat, o[u] - (k0 + stride * u)) ^ load8(txt, o[u])) : 0;
        any = false;
#pragma unroll
        for (int u = 0; u < N; ++u) {
            if (!run[u]) continue;
            if (x[u]) {
                o[u] += (__ffsll((long long)x[u]) - 1) >> 3;
                run[u] = false;
            } else {
                o[u] += 8;
                any = true;
            }
        }
    }
}

// The result of one pair (one thread): the backtrace of a pair that reached the end
// (status 0), the CIGAR operations reversed into forward order, and the output record.
template <bool PIG>
__device__ void finish_pair(const WfaArgs &A, const WfaPairDev &PR, int idx, const uint8_t *pat, const uint8_t *txt,
                            const int64_t *ctab, const HdrRing &HR, int status, int end_score, int s, int64_t used) {
    const WfaPen P = A.pen;
    const int plen = PR.plen, tlen = PR.tlen;
    const int k_end = tlen - plen;
    WfaOutDev o;
    o.status = status, o.score = 0, o.n_ops = 0, o.final_s = s;
    o.mem_bytes = used;
    if (status == 0) {
        OpsWriter w{A.ops + PR.ops_off, 0, plen + tlen + 8, true};
        if constexpr (PIG) {
            // reverse the links from the end cell in place, then unpack the blocks
            // oldest first: before every operation taken in M the run of matches
            // is re-extended; the mismatch that closes a gap is dropped
            const CompHdr m = HR.get(A, ctab, CM, end_score);
            const uint32_t *md = (const uint32_t *)(A.pool + m.off) + (k_end - m.base);
            const uint32_t pc_end = md[m.pad];
            uint32_t cur = md[2 * m.pad], prv = BT_NULL;
            uint2 *blk = (uint2 *)A.pool;
            const int64_t lim = 2 * ((int64_t)plen + tlen) + 64;
            int64_t steps = 0;
            bool ok = true;
            while (cur != BT_NULL) {
                if (++steps > lim) { ok = false; break; }
                const uint32_t nxt = blk[cur].y;
                blk[cur].y = prv;
                prv = cur, cur = nxt;
            }
            int64_t v = 0, h = 0;
            bool in_m = true;
            cur = prv;
            for (bool last = false; ok && !last;) {
                uint32_t pc;
                if (cur != BT_NULL) pc = blk[cur].x, cur = blk[cur].y;
                else pc = pc_end, last = true;
                const int len = pc ? 16 - (__clz(pc) >> 1) : 0;
                for (int j = len - 1; j >= 0; --j) {
                    if (in_m) {
                        const int64_t nm = lcp1(A, PR, pat, txt, v, h);
                        w.put('M', (int)nm);
                        v += nm, h += nm;
                    }
                    const uint32_t op = (pc >> (2 * j)) & 3u;
                    if (!in_m && op == 2u) {
                        in_m = true;
                        continue;
                    }
                    w.put(op == 1u ? 'D' : op == 2u ? 'X' : 'I', 1);
                    v += (op == 1u || op == 2u), h += (op == 2u || op == 3u);
                    in_m = op == 2u;
                    if (op == 0u || v > plen || h > tlen) { ok = false; break; }
                }
            }
            if (ok) {
                const int64_t nm = min((int64_t)plen - v, (int64_t)tlen - h);
                w.put('M', (int)nm);
                v += nm, h += nm;
                w.put('I', (int)(tlen - h));
                w.put('D', (int)(plen - v));
            } else {
                o.status = WFA_UNATTAINABLE;
            }
        } else if (!A.singletrack) {
            enum { BM = 9, BD2E = 8, BD2O = 7, BD1E = 6, BD1O = 5, BI2E = 4, BI2O = 3, BI1E = 2, BI1O = 1 };
            int mt = CM, sc = end_score, k = k_end;
            int32_t off = tlen;
            int v = off - k, h = off;
            const int64_t NEG = pb(WF_NULL, 0);
            while (v > 0 && h > 0 && sc > 0) {
                const int smm = sc - P.x, sg1 = sc - P.o1 - P.e1, sg2 = sc - P.o2 - P.e2, sx1 = sc - P.e1,
                          sx2 = sc - P.e2;
                auto G = [&](int scr, int comp, int kk, int add, int t) -> int64_t {
                    if (scr < 0) return NEG;
                    const CompHdr hh = hdr_ptr(A, ctab, scr)->c[comp];
                    return pb(getv(A, hh, kk) + add, t);
                };
                int64_t mall;
                const int64_t i1o = (mt == CM || mt == CI1) ? G(sg1, CM, k - 1, 1, BI1O) : NEG;
                const int64_t i1e = (mt == CM || mt == CI1) ? G(sx1, CI1, k - 1, 1, BI1E) : NEG;
                const int64_t d1o = (mt == CM || mt == CD1) ? G(sg1, CM, k + 1, 0, BD1O) : NEG;
                const int64_t d1e = (mt == CM || mt == CD1) ? G(sx1, CD1, k + 1, 0, BD1E) : NEG;
                const int64_t i2o = (mt == CM || mt == CI2) ? G(sg2, CM, k - 1, 1, BI2O) : NEG;
                const int64_t i2e = (mt == CM || mt == CI2) ? G(sx2, CI2, k - 1, 1, BI2E) : NEG;
                const int64_t d2o = (mt == CM || mt == CD2) ? G(sg2, CM, k + 1, 0, BD2O) : NEG;
                const int64_t d2e = (mt == CM || mt == CD2) ? G(sx2, CD2, k + 1, 0, BD2E) : NEG;
                if (mt == CM) {
                    const int64_t misms = G(smm, CM, k, 1, BM);
                    mall = max(misms, max(max(max(i1o, i1e), max(i2o, i2e)), max(max(d1o, d1e), max(d2o, d2e))));
                } else if (mt == CI1) mall = max(i1o, i1e);
                else if (mt == CI2) mall = max(i2o, i2e);
                else if (mt == CD1) mall = max(d1o, d1e);
                else mall = max(d2o, d2e);
                if (mall < 0) break;
                if (mt == CM) {
                    const int mo = (int)(mall >> 4);
                    w.put('M', off - mo);
                    off = mo;
                    v = off - k, h = off;
                    if (v <= 0 || h <= 0) break;
                }
                const int bt = (int)(mall & 0xf);
                switch (bt) {
                case BM: sc = smm; mt = CM; break;
                case BI1O: sc = sg1; mt = CM; break;
                case BI1E: sc = sx1; mt = CI1; break;
                case BI2O: sc = sg2; mt = CM; break;
                case BI2E: sc = sx2; mt = CI2; break;
                case BD1O: sc = sg1; mt = CM; break;
                case BD1E: sc = sx1; mt = CD1; break;
                case BD2O: sc = sg2; mt = CM; break;
                default: sc = sx2; mt = CD2; break;
                }
                if (bt == BM) w.put('X', 1), --off;
                else if (bt <= BI2E) w.put('I', 1), --k, --off;
                else w.put('D', 1), ++k;
                v = off - k, h = off;
            }
            if (mt == CM) {
                if (v > 0 && h > 0) {
                    const int nm = v < h ? v : h;
                    w.put('M', nm);
                    v -= nm, h -= nm;
                }
                w.put('D', v > 0 ? v : 0);
                w.put('I', h > 0 ? h : 0);
            }
        } else {
            int sc = end_score, k = k_end, gl = 0;
            bool in_m = true, ok = true;
            int32_t off = tlen, off_be = off;
            const int64_t maxgap = (int64_t)plen + tlen;
            while (sc != 0) {
                if (sc < 0 || off < 0) { ok = false; break; }
                if (in_m) {
                    const int v = off - k, h = off;
                    if (v < 0 || h < 0 || v > plen || h > tlen) { ok = false; break; }
                    int nm = 0;
                    while (nm < v && nm < h && pat[v - nm - 1] == txt[h - nm - 1]) ++nm;
                    off_be = off - nm;
                    const int ms = sc - P.x;
                    bool took = false;
                    if (ms >= 0) {
                        const CompHdr mh = hdr_ptr(A, ctab, ms)->c[CM];
                        if (mh.lo <= k && k <= mh.hi &&
                            ((const int32_t *)(A.pool + mh.off))[k - mh.base] + 1 == off_be) {
                            w.put('M', nm);
                            w.put('X', 1);
                            off = off_be - 1;
                            sc = ms;
                            took = true;
                        }
                    }
                    if (!took) in_m = false, gl = 0;
                    continue;
                }
                ++gl;
                if ((int64_t)gl > maxgap) { ok = false; break; }
                const int ki = k - gl, kd = k + gl;
                for (int piece = 0; piece < 2; ++piece) {
                    const int64_t isc = piece == 0 ? (int64_t)sc - P.o1 - (int64_t)gl * P.e1
                                                   : (int64_t)sc - P.o2 - (int64_t)gl * P.e2;
                    if (isc < 0 || isc > s) continue;
                    const CompHdr ih = hdr_ptr(A, ctab, (int)isc)->c[CM];
                    const int32_t *id = (const int32_t *)(A.pool + ih.off);
                    if (ih.lo <= ki && ki <= ih.hi && id[ki - ih.base] + gl >= off_be &&
                        id[ki - ih.base] + gl <= off) {
                        w.put('M', off - (id[ki - ih.base] + gl));
                        w.put('I', gl);
                        k = ki, off = id[ki - ih.base], sc = (int)isc, in_m = true;
                        break;
                    }
                    if (ih.lo <= kd && kd <= ih.hi && id[kd - ih.base] >= off_be && id[kd - ih.base] <= off) {
                        w.put('M', off - id[kd - ih.base]);
                        w.put('D', gl);
                        k = kd, off = id[kd - ih.base], sc = (int)isc, in_m = true;
                        break;
                    }
                }
            }
            if (ok && (!in_m || k != 0 || off < 0 || off > plen || off > tlen)) ok = false;
            if (ok)
                for (int i = 0; i < off; ++i)
                    if (pat[i] != txt[i]) { ok = false; break; }
            if (ok) w.put('M', off);
            if (!ok) o.status = WFA_UNATTAINABLE;
        }
        if (!w.ok) o.status = WFA_OVERFLOW;
        if (o.status == 0) {
            for (int a = 0, b = PIG ? 0 : w.n - 1; a < b; ++a, --b) {
                const char t = w.buf[a];
                w.buf[a] = w.buf[b], w.buf[b] = t;
            }
            o.score = -end_score;
            o.n_ops = w.n;
        }
    }
    A.out[idx] = o;
}

// One trip of the piggyback compute step over the diagonals kb + g0 + G*u (u < PIG_U) of a
// score with range [lo, hi], inputs in[] (M[s-x], M[s-o1-e1], I1[s-e1], D1[s-e1], M[s-o2-e2],
// I2[s-e2], D2[s-e2]) and outputs out[] (ring slots of rcap elements per array).  Each gap cell
// takes the extension on a tie, M the mismatch, then D2, D1, I2, I1 (the kernel's assignment
// order); M is extended as it is computed (matches are not recorded in the packed CIGAR; the
// traceback re-extends them).  Cells whose packed CIGAR holds 15 operations move it into a
// block from the lane's reserved run; lanes whose run is short reserve LANE_BLOCKS more in one
// allocation of the warp (`wal`).  Every lane of the warp must call it.  Returns false when
// the pool is exhausted.
template <bool TRIM = true>
__device__ __forceinline__ bool pig_trip(const WfaArgs &A, const WfaPairDev &PR, const uint8_t *pat,
                                         const uint8_t *txt, int kb, int g0, int G, int lo, int hi,
                                         const CompHdr (&in)[7], const CompHdr (&out)[5], int mask, int rcap,
                                         Alloc &wal, uint32_t &bnext, uint32_t &bend, int (&kmin)[5], int (&kmax)[5],
                                         bool &reached, bool &beyond) {
    const int plen = PR.plen, tlen = PR.tlen, k_end = tlen - plen, lane = threadIdx.x & 31;
    const CompHdr &m_misms = in[0], &m_open1 = in[1], &i1 = in[2], &d1 = in[3], &m_open2 = in[4], &i2 = in[5],
                  &d2 = in[6];
    const int k0 = kb + g0;
    Cell C[PIG_U][5];
#pragma unroll
    for (int u = 0; u < PIG_U; ++u) {
        const int k = k0 + G * u;
        Cell a = getc(A, m_open1, k - 1), b = getc(A, i1, k - 1);
        Cell g = b.o >= a.o ? b : a;
        C[u][CI1] = Cell{g.o + 1, (g.pc << 2) | 3u, g.pv};
        a = getc(A, m_open2, k - 1), b = getc(A, i2, k - 1);
        g = b.o >= a.o ? b : a;
        C[u][CI2] = Cell{g.o + 1, (g.pc << 2) | 3u, g.pv};
        a = getc(A, m_open1, k + 1), b = getc(A, d1, k + 1);
        g = b.o >= a.o ? b : a;
        C[u][CD1] = Cell{g.o, (g.pc << 2) | 1u, g.pv};
        a = getc(A, m_open2, k + 1), b = getc(A, d2, k + 1);
        g = b.o >= a.o ? b : a;
        C[u][CD2] = Cell{g.o, (g.pc << 2) | 1u, g.pv};
        Cell x = getc(A, m_misms, k);
        x.o += 1;
        const int32_t best = max(max(C[u][CD1].o, C[u][CD2].o), max(x.o, max(C[u][CI1].o, C[u][CI2].o)));
        const Cell &src = best == x.o ? x
                          : best == C[u][CD2].o ? C[u][CD2]
                          : best == C[u][CD1].o ? C[u][CD1]
                          : best == C[u][CI2].o ? C[u][CI2]
                                                : C[u][CI1];
        C[u][CM] = Cell{in_matrix(best, k, plen, tlen) ? best : WF_NULL, (src.pc << 2) | 2u, src.pv};
        const int32_t gap = max(max(C[u][CD1].o, C[u][CD2].o), max(C[u][CI1].o, C[u][CI2].o));
        if (k <= hi && gap >= 0 && gap > min(tlen, k + plen)) beyond = true;
    }
    {
        int32_t mo[PIG_U];
#pragma unroll
        for (int u = 0; u < PIG_U; ++u) mo[u] = k0 + G * u <= hi ? C[u][CM].o : WF_NULL;
        extend_n<PIG_U>(PR, bases_of(A, PR), pat, txt, k0, G, mo);
#pragma unroll
        for (int u = 0; u < PIG_U; ++u) {
            const int k = k0 + G * u;
            if (k > hi) continue;
            C[u][CM].o = mo[u];
            if (k == k_end && mo[u] != WF_NULL && mo[u] >= tlen) reached = true;
        }
    }
    uint32_t fl = 0;
#pragma unroll
    for (int u = 0; u < PIG_U; ++u) {
        const int k = k0 + G * u;
#pragma unroll
        for (int c = 0; c < 5; ++c)
            if (k <= hi && (mask & (1 << c)) && C[u][c].pc >= PC_ALMOST_FULL && in_matrix(C[u][c].o, k, plen, tlen))
                fl |= 1u << (u * 5 + c);
    }
    const bool refill = bend - bnext < (uint32_t)__popc(fl);
    const unsigned rb = __ballot_sync(0xffffffffu, refill);
    if (rb) {
        const int64_t bb = warp_alloc(A, wal, (int64_t)__popc(rb) * LANE_BLOCKS * 8, lane);
        if (bb < 0) return false;
        if (refill) {
            bnext = (uint32_t)(bb >> 3) + (uint32_t)__popc(rb & ((1u << lane) - 1u)) * LANE_BLOCKS;
            bend = bnext + LANE_BLOCKS;
        }
    }
    if (fl) {
        uint2 *blk = (uint2 *)A.pool;
#pragma unroll
        for (int u = 0; u < PIG_U; ++u)
#pragma unroll
            for (int c = 0; c < 5; ++c)
                if (fl & (1u << (u * 5 + c))) {
                    blk[bnext] = make_uint2(C[u][c].pc, C[u][c].pv);
                    C[u][c].pc = 0u, C[u][c].pv = bnext++;
                }
    }
#pragma unroll
    for (int u = 0; u < PIG_U; ++u) {
        const int k = k0 + G * u;
        if (k > hi) break;
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            if (!(mask & (1 << c))) continue;
            int32_t *d = (int32_t *)(A.pool + out[c].off) + (k - lo);
            d[0] = C[u][c].o, d[rcap] = (int32_t)C[u][c].pc, d[2 * rcap] = (int32_t)C[u][c].pv;
            if (TRIM && in_matrix(C[u][c].o, k, plen, tlen)) kmin[c] = min(kmin[c], k), kmax[c] = max(kmax[c], k);
        }
    }
    return true;
}

// ---------------------------------------------------------------------------------------
// Plans and partials shared by the CTA-cooperative mode below and the cluster kernel: the
// plan of one score (its range, inputs and outputs) and, per CTA, the trimmed ends of each
// component and whether the end cell was reached.
enum { WOP_COMPUTE = 0, WOP_DONE = 1, WOP_EXIT = 2 };

struct WidePlan {
    int op, lo, hi, mask;  // mask: components allocated at the planned score (bit c)
    int ilo, ihi;          // the diagonals that every input has; ilo > ihi unless mask is full
    int s;                 // the planned score (cluster kernel)
    CompHdr in[7];         // M[s-x], M[s-o1-e1], I1[s-e1], D1[s-e1], M[s-o2-e2], I2[s-e2], D2[s-e2]
    CompHdr out[5];
    InHdr view[7];         // the same inputs as the compute step of the high memory modes reads them
    int32_t *dst[5];       // and where it writes diagonal lo (null: not stored)
};
// Maxima over a CTA's diagonals, folded by atomicMax: k[c] the highest diagonal of component
// c in the matrix, k[5 + c] minus the lowest, k[10] 1 when the end cell was reached.
struct __align__(16) WidePart {
    int k[12];
    int pad[2];
    unsigned long long used;  // bytes of the warps' block reservations (CTA-cooperative piggyback mode)
};

__device__ __forceinline__ void part_reset(WidePart &p, int lane) {
    if (lane < 12) p.k[lane] = INT_MIN;
}

// Planning a score takes one warp: lane j < 7 holds the j-th input of the compute step (M[s-x],
// M[s-o1-e1], I1[s-e1], D1[s-e1], M[s-o2-e2], I2[s-e2], D2[s-e2]): its component, its distance
// in scores, and how it moves the limits.  A null input contributes lo=1, hi=-1.
struct PlanLane {
    int comp, dist, dlo, dhi;
};
__device__ __forceinline__ PlanLane plan_lane(const WfaPen &P, int lane) {
    switch (lane) {
    case 0: return PlanLane{CM, P.x, 0, 0};
    case 1: return PlanLane{CM, P.o1 + P.e1, -1, 1};
    case 2: return PlanLane{CI1, P.e1, 1, 1};
    case 3: return PlanLane{CD1, P.e1, -1, -1};
    case 4: return PlanLane{CM, P.o2 + P.e2, -1, 1};
    case 5: return PlanLane{CI2, P.e2, 1, 1};
    case 6: return PlanLane{CD2, P.e2, -1, -1};
    default: return PlanLane{CM, 0, 0, 0};
    }
}
// The limits of the compute step and which I/D outputs exist (one of their inputs exists).
__device__ __forceinline__ void plan_limits(const PlanLane &L, int lane, const CompHdr &h, unsigned some, int &lo, int &hi,
                                            int &mask) {
    lo = __reduce_min_sync(0xffffffffu, lane < 7 ? h.lo + L.dlo : INT_MAX);
    hi = __reduce_max_sync(0xffffffffu, lane < 7 ? h.hi + L.dhi : INT_MIN);
    mask = 1;
    if (some & (1u << 1 | 1u << 2)) mask |= 1 << CI1;
    if (some & (1u << 1 | 1u << 3)) mask |= 1 << CD1;
    if (some & (1u << 4 | 1u << 5)) mask |= 1 << CI2;
    if (some & (1u << 4 | 1u << 6)) mask |= 1 << CD2;
}

// The diagonals that all seven inputs have, if every component is an output.
__device__ __forceinline__ void plan_inner(WidePlan &q, int mask, int lane, const CompHdr &h) {
    const int ilo = __reduce_max_sync(0xffffffffu, lane < 7 ? h.lo : INT_MIN);
    const int ihi = __reduce_min_sync(0xffffffffu, lane < 7 ? h.hi : INT_MAX);
    if (lane == 0) q.ilo = ilo, q.ihi = mask == 31 ? ihi : ilo - 1;
}

// A warp's trimmed ends and end check, folded into its CTA's partials.
__device__ __forceinline__ void fold_partials(const int (&kmin)[5], const int (&kmax)[5], bool reached, WidePart &pp) {
    const int lane = threadIdx.x & 31;
    int v = __any_sync(0xffffffffu, reached) ? 1 : INT_MIN;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const int th = __reduce_max_sync(0xffffffffu, kmax[c]);
        const int tl = __reduce_max_sync(0xffffffffu, -kmin[c]);
        if (lane == c) v = th;
        if (lane == 5 + c) v = tl;
    }
    if (lane < 11 && v != INT_MIN) atomicMax(&pp.k[lane], v);
}

// First array of component c at score sc in the piggyback rings: M's last SR scores, then
// I1/D1's last R1, then I2/D2's last R2, three arrays (offsets, packed CIGARs, links) each.
__device__ __forceinline__ int64_t pig_slot(int c, int sc, int SR, int R1, int R2) {
    if (c == CM) return (int64_t)(sc % SR) * 3;
    if (c <= CD1) return 3 * (int64_t)(SR + (sc % R1) * 2 + (c - CI1));
    return 3 * (int64_t)(SR + 2 * R1 + (sc % R2) * 2 + (c - CI2));
}

// Diagonals per thread in flight in the CTA-cooperative compute step (build-time tuning).
#ifndef AW_WFA_CTA_U
#define AW_WFA_CTA_U 2
#endif

// U diagonals k0 + G*u <= hi of one thread (high memory): the compute step, the fused extension
// of M, the stores, this thread's trimmed ends (TRIM), and whether it met the end cell or an
// offset beyond the end of a sequence.  v: the inputs; dst[c]: where component c's diagonal lo
// goes (null: nowhere).  INNER: every input has the diagonals k-1 .. k+1, and all components are
// stored; without GUARD no k is beyond hi either.  A trip is bound by its instructions and
// their latencies (few warps per SM): G is known at build time so that a trip's diagonals
// differ by an immediate, and as a real offset is never negative, nor before the start of a
// sequence, one compare with the diagonal's length puts an offset inside the matrix.
template <int U, int G, bool INNER, bool GUARD, bool TRIM, bool SH>
__device__ __forceinline__ void wf_trip(const WfaPairDev &PR, const Bases &B, const uint8_t *pat, const uint8_t *txt,
                                        const InHdr (&v)[7], int32_t *const (&dst)[5], int lo, int hi, int k0,
                                        int (&kmin)[5], int (&kmax)[5], bool &reached, bool &beyond) {
    int32_t g[U][4], misms[U], mo[U];  // I1, D1, I2, D2
    int32_t *to[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) to[c] = INNER || dst[c] ? dst[c] + (k0 - lo) : nullptr;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k = k0 + G * u;
        auto in = [&](int j, int d) -> int32_t {
            if constexpr (!INNER) return getv(v[j], k + d);
            else return !GUARD || k <= hi ? (v[j].p + k0)[G * u + d] : WF_NULL;
        };
        g[u][0] = max(in(1, -1), in(2, -1)) + 1;
        g[u][1] = max(in(1, 1), in(3, 1));
        g[u][2] = max(in(4, -1), in(5, -1)) + 1;
        g[u][3] = max(in(4, 1), in(6, 1));
        misms[u] = in(0, 0) + 1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k = k0 + G * u;
        const bool here = !GUARD || k <= hi;
        // offsets 0 .. lim - 1 lie in the matrix
        const uint32_t lim = here ? (uint32_t)max(min(PR.tlen, k + PR.plen) + 1, 0) : 0u;
        const int32_t gap = max(max(g[u][0], g[u][1]), max(g[u][2], g[u][3]));
        const int32_t best = max(gap, misms[u]);
        mo[u] = (uint32_t)best < lim ? best : WF_NULL;
        if (here && gap >= (int32_t)lim) beyond = true;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (here && (INNER || to[c + 1])) to[c + 1][G * u] = g[u][c];
            if (TRIM && (uint32_t)g[u][c] < lim) kmin[c + 1] = min(kmin[c + 1], k), kmax[c + 1] = max(kmax[c + 1], k);
        }
        if (TRIM && (uint32_t)best < lim) kmin[CM] = min(kmin[CM], k), kmax[CM] = max(kmax[CM], k);
    }
    extend_n<U, SH>(PR, B, pat, txt, k0, G, mo);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k = k0 + G * u;
        if (GUARD && k > hi) break;
        if (k == PR.tlen - PR.plen && mo[u] >= PR.tlen) reached = true;
        to[CM][G * u] = mo[u];
    }
}

// The trip whose first lane has diagonal kw, with or without checks.
template <int U, int G, bool SH, bool TRIM>
__device__ __forceinline__ void plan_trip(const WfaPairDev &PR, const Bases &B, const uint8_t *pat, const uint8_t *txt,
                                          const WidePlan &Q, int kw, int lane, int (&kmin)[5], int (&kmax)[5],
                                          bool &reached, bool &beyond) {
    if (kw > Q.ilo && kw + 31 + G * (U - 1) < Q.ihi)
        wf_trip<U, G, true, false, TRIM, SH>(PR, B, pat, txt, Q.view, Q.dst, Q.lo, Q.hi, kw + lane, kmin, kmax, reached, beyond);
    else if (kw <= Q.hi)
        wf_trip<U, G, false, true, TRIM, SH>(PR, B, pat, txt, Q.view, Q.dst, Q.lo, Q.hi, kw + lane, kmin, kmax, reached, beyond);
}

// The diagonals of a planned score (high memory) of one warp of CTA `rank` of CL, each CTA with G
// computing threads, folded into the CTA's partials.  The wavefront is taken in rounds of
// CL*G*U diagonals, with the fewest diagonals per thread that end it: narrow ones are spread over
// all threads.  Returns, for the warp, 1 when the end cell was reached, plus 2 when a gap
// component got an offset beyond the end of a sequence.
template <int UMAX, int G, bool SH, bool TRIM = true>
__device__ __forceinline__ int plan_compute(const WfaPairDev &PR, const Bases &B, const uint8_t *pat,
                                            const uint8_t *txt, const WidePlan &Q, int rank, int CL, WidePart &pp) {
    const int lane = threadIdx.x & 31, w0 = threadIdx.x & ~31;
    int kmin[5], kmax[5];
    bool reached = false, beyond = false, any = false;
#pragma unroll
    for (int c = 0; c < 5; ++c) kmin[c] = INT_MAX, kmax[c] = INT_MIN;
    for (int kb = Q.lo; kb <= Q.hi;) {
        const int left = Q.hi - kb + 1, round = CL * G;
        const int U = UMAX >= 4 && left > 2 * round ? 4 : UMAX >= 2 && left > round ? 2 : 1;
        const int kw = kb + rank * G * U + w0;
        any |= kw <= Q.hi;
        if (UMAX >= 4 && U == 4) plan_trip<4, G, SH, TRIM>(PR, B, pat, txt, Q, kw, lane, kmin, kmax, reached, beyond);
        else if (UMAX >= 2 && U == 2) plan_trip<2, G, SH, TRIM>(PR, B, pat, txt, Q, kw, lane, kmin, kmax, reached, beyond);
        else plan_trip<1, G, SH, TRIM>(PR, B, pat, txt, Q, kw, lane, kmin, kmax, reached, beyond);
        kb += round * U;
    }
    if (!any) return 0;  // no diagonal for this warp
    if (TRIM) fold_partials(kmin, kmax, reached, pp);
    return (__any_sync(0xffffffffu, reached) ? 1 : 0) | (__any_sync(0xffffffffu, beyond) ? 2 : 0);
}

// The same without trimmed ends, for the cluster kernel's CTAs of G + 32 computing threads: G of
// them take the diagonals that every input has; the few on either side, with their checks, are
// the work of the last warp of the first and of the last CTA.
template <int G, bool SH>
__device__ __forceinline__ int plan_open(const WfaPairDev &PR, const Bases &B, const uint8_t *pat, const uint8_t *txt,
                                         const WidePlan &Q, int rank, int CL) {
    const int lane = threadIdx.x & 31, w0 = threadIdx.x & ~31;
    int kmin[5], kmax[5];  // not used
    bool reached = false, beyond = false;
    const int first = Q.ilo + 1, last = Q.ihi - 1;
    if (last - first < 64) {
        for (int kw = Q.lo + rank * (G + 32) + w0; kw <= Q.hi; kw += CL * (G + 32))
            wf_trip<1, G, false, true, false, SH>(PR, B, pat, txt, Q.view, Q.dst, Q.lo, Q.hi, kw + lane, kmin, kmax,
                                                  reached, beyond);
    } else if (w0 == G) {
        for (int side = 0; side < 2; ++side) {
            if (rank != (side ? CL - 1 : 0)) continue;
            const int end = side ? Q.hi : first - 1;
            for (int kw = side ? last + 1 : Q.lo; kw <= end; kw += 32)
                wf_trip<1, G, false, true, false, SH>(PR, B, pat, txt, Q.view, Q.dst, Q.lo, end, kw + lane, kmin, kmax,
                                                      reached, beyond);
        }
    } else {
        for (int kb = first; kb <= last;) {
            const int left = last - kb + 1, round = CL * G;
            const int U = left > 2 * round ? 4 : left > round ? 2 : 1;
            const int kw = kb + rank * G * U + w0;
            if (kw > last) break;
            if (U == 4)
                wf_trip<4, G, true, true, false, SH>(PR, B, pat, txt, Q.view, Q.dst, Q.lo, last, kw + lane, kmin, kmax,
                                                     reached, beyond);
            else if (U == 2)
                wf_trip<2, G, true, true, false, SH>(PR, B, pat, txt, Q.view, Q.dst, Q.lo, last, kw + lane, kmin, kmax,
                                                     reached, beyond);
            else
                wf_trip<1, G, true, true, false, SH>(PR, B, pat, txt, Q.view, Q.dst, Q.lo, last, kw + lane, kmin, kmax,
                                                     reached, beyond);
            kb += round * U;
        }
    }
    return (__any_sync(0xffffffffu, reached) ? 1 : 0) | (__any_sync(0xffffffffu, beyond) ? 2 : 0);
}

// The trimmed ends of a computed score, from its stored offsets, folded into the CTA's partials.
__device__ __noinline__ void plan_trim(const WfaPairDev &PR, const WidePlan &Q, int g0, int G, WidePart &pp) {
    int kmin[5], kmax[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) kmin[c] = INT_MAX, kmax[c] = INT_MIN;
    for (int k = Q.lo + g0; k <= Q.hi; k += G) {
#pragma unroll
        for (int c = 0; c < 5; ++c)
            if (Q.dst[c] && in_matrix(Q.dst[c][k - Q.lo], k, PR.plen, PR.tlen)) kmin[c] = min(kmin[c], k), kmax[c] = max(kmax[c], k);
    }
    __syncwarp();
    fold_partials(kmin, kmax, false, pp);
}

// CTA-cooperative mode: one long pair on a CTA of NT computing threads and one planning warp.  As in
// the cluster kernel (below), wavefronts are not trimmed before the first offset beyond the end of a sequence, so that the planner works a score ahead of the others and one
// CTA barrier per score is left (two, with the plan between them, took 3.8 us a score at 2 kb,
// half of it waiting for the plan; now 2.3).  A pair whose wavefront grows too wide stops with
// WFA_WIDE for the cluster kernel; in the piggyback modes none does, and every warp reserves its own
// block runs.  A pair that takes the last of the pool (WfaArgs::free_slots) is trimmed from the start.
struct CtaShared {
    WidePlan plan[2];
    WidePart part;
    // flags of step it at it % 3 (a fast warp may set those of step it + 1 before a slow one has
    // read step it's); retry: a warp found the pool exhausted
    int at_end[3], beyond[3], retry[3];
    int next;  // position of the pair
};
template <bool PIG, int NT>
__device__ void cta_open(const WfaArgs &A, int idx, const HdrRing &HR, CtaShared &S, Alloc &al) {
    const int tid = threadIdx.x, lane = tid & 31;
    const bool planner = tid >= NT;
    const WfaPen P = A.pen;
    const WfaPairDev PR = A.pairs[idx];
    const int plen = PR.plen, tlen = PR.tlen;
    const uint8_t *pat = A.pat + PR.poff, *txt = A.txt + PR.toff;
    const Bases B = bases_of(A, PR);
    int64_t *ctab = A.ctab + PR.ctab_off;
    const CompHdr NUL{1, -1, 0, 0, 0};
    const int smax = PR.ctab_cap * HDR_CHUNK - 1;
    const int R = (P.e1 > P.e2 ? P.e1 : P.e2) + 1, ring_cap = plen + tlen + 8;
    const PlanLane L = plan_lane(P, lane);
    // where this lane of the planner reads its input and writes its component (no rings: the
    // pool).  Kept for the high-memory planner only, which bounds a score of short wavefronts (4,096
    // pairs 33.3 -> 32.4 ms, 16,384 103 -> 96); the piggyback trips need the registers.
    const bool rings = !PIG && HR.sh.mm >= 0;
    const CompHdr *const rd = rings ? HR.at(L.comp, 0) : nullptr;
    CompHdr *const wr = rings ? HR.at(min(lane, 4), 0) : nullptr;
    const int rd_mask = HR.mask(L.comp), wr_mask = HR.mask(min(lane, 4));
    // the planner's place in its chunk, the same in all lanes
    int64_t cur = 0, chunk_end = 0;
    auto alloc = [&](int64_t bytes) -> int64_t {
        if constexpr (PIG) return warp_alloc(A, al, bytes, lane);
        bytes = (bytes + 15) & ~(int64_t)15;
        if (cur + bytes > chunk_end) {
            if (lane == 0) al.cur = cur;
            int ok = lane == 0 ? take_chunk(pool_of(A), al, bytes) : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) return -1;
            __syncwarp();
            cur = al.cur, chunk_end = al.end;
        }
        const int64_t r = cur;
        cur += bytes;
        return r;
    };
    // the planner's state: the planned score, the last one with headers, the header chunk of the
    // scores from s_hdr on, the planned score's header of component `lane`
    int s = 0, committed = 0, num_null = 0, status = 0, end_score = -1, s_hdr = 0, slot = 0;
    int64_t ring = -1, hdr_off = 0;
    CompHdr mine = NUL;
    // piggyback: the rings' place and the elements of a slot's array, every warp's block run
    const int SR = A.max_score_scope, R1 = P.e1 + 1, R2 = P.e2 + 1;
    const int64_t ring_arrays = 3 * (int64_t)(SR + 2 * R1 + 2 * R2);
    int rcap = 32;
    uint32_t bnext = 0, bend = 0;
    if (PIG && !planner && lane == 0) al.init();
    auto set_hdr = [&](int sc, const CompHdr &o) {
        if (lane < 5) {
            const int64_t off = sc >= s_hdr ? hdr_off : ctab[sc / HDR_CHUNK];
            ((ScoreHdr *)(A.pool + off))[sc % HDR_CHUNK].c[lane] = o;
            if (rings) wr[sc & wr_mask] = o;
            else HR.put(lane, sc, o);
        }
        __syncwarp();
    };
    // the headers of score sc, and of the null scores before it
    auto commit = [&](int sc, const CompHdr &o) {
        for (int z = committed + 1; z < sc; ++z) set_hdr(z, NUL);
        set_hdr(sc, o);
        committed = sc;
    };
    auto plan_next = [&](WidePlan &q) {
        for (;;) {
            ++s;
            slot = slot + 1 == R ? 0 : slot + 1;
            if (s > smax) {
                status = WFA_OVERFLOW;
                break;
            }
            if (s % HDR_CHUNK == 0) {
                const int64_t hb = alloc((int64_t)sizeof(ScoreHdr) * HDR_CHUNK);
                if (hb < 0) {
                    status = WFA_RETRY;
                    break;
                }
                hdr_off = hb, s_hdr = s;
                if (lane == 0) ctab[s / HDR_CHUNK] = hb;
                __syncwarp();
            }
            // the scores since the last committed one are null
            CompHdr in = NUL;
            if (lane < 7 && s - L.dist >= 0 && s - L.dist <= committed) in = rings ? rd[(s - L.dist) & rd_mask] : HR.get(A, ctab, L.comp, s - L.dist);
            const unsigned some = __ballot_sync(0xffffffffu, lane < 7 && in.lo <= in.hi);
            if (!some) {
                if (++num_null > A.max_score_scope) {  // the top of the next step: M[s] is empty
                    status = -3;
                    break;
                }
                continue;
            }
            num_null = 0;
            int lo, hi, mask;
            plan_limits(L, lane, in, some, lo, hi, mask);
            // no diagonal beyond these has a cell
            lo = max(lo, -plen), hi = min(hi, tlen);
            const int width = hi - lo + 1;
            if constexpr (PIG) {
                if (width > rcap) {
                    const int nc = max(2 * rcap, (width + 3) & ~3);
                    const int64_t nb = alloc(ring_arrays * nc * 4);
                    if (nb < 0) {
                        status = WFA_RETRY;
                        break;
                    }
                    rcap = nc, ring = nb;
                }
                if (lane < 5) {
                    mine = mask >> lane & 1
                               ? CompHdr{lo, hi, lo, rcap, ring + pig_slot(lane, s, SR, R1, R2) * rcap * 4}
                               : NUL;
                    q.out[lane] = mine;
                    q.dst[lane] = mask >> lane & 1 ? (int32_t *)(A.pool + mine.off) : nullptr;
                }
                if (lane < 7) q.in[lane] = in;
                if (lane == 0) q.op = WOP_COMPUTE, q.lo = lo, q.hi = hi, q.mask = mask, q.s = s;
                __syncwarp();
                return;
            }
            // a wavefront too wide for the CTA: the cluster kernel re-runs the pair (past
            // wide_width_cta always; past wide_tail_cta in the call's tail, checked every 32
            // scores: every pair started and few still running)
            if (A.wide_width_cta > 0 && width > A.wide_tail_cta) {
                bool wide = width > A.wide_width_cta;
                if (!wide && (s & 31) == 0)
                    wide = __all_sync(0xffffffffu, *(volatile int32_t *)(A.queue + 3) >= A.n_all &&
                                                       *(volatile int32_t *)(A.queue + 1) <= A.wide_tail_pairs);
                if (wide) {
                    status = WFA_WIDE;
                    break;
                }
            }
            if (A.singletrack && width > ring_cap) {
                status = WFA_OVERFLOW;
                break;
            }
            const int64_t wb = (((int64_t)width * 4) + 15) & ~(int64_t)15;
            const int64_t blk = alloc(wb * (A.singletrack ? 1 : __popc(mask)));
            if (blk < 0) {
                status = WFA_RETRY;
                break;
            }
            if (lane < 5) {
                mine = NUL;
                if (mask >> lane & 1)
                    mine = CompHdr{lo, hi, lo, 0,
                                   lane == CM || !A.singletrack ? blk + wb * __popc(mask & ((1 << lane) - 1))
                                                                : ring + ((int64_t)(slot * 4 + (lane - 1)) * ring_cap) * 4};
                q.out[lane] = mine;
                q.dst[lane] = mask >> lane & 1 ? (int32_t *)(A.pool + mine.off) : nullptr;
            }
            if (lane < 7) q.view[lane] = in_hdr(A, in);
            plan_inner(q, mask, lane, in);
            if (lane == 0) q.op = WOP_COMPUTE, q.lo = lo, q.hi = hi, q.mask = mask, q.s = s;
            __syncwarp();
            return;
        }
        if (lane == 0) q.op = WOP_DONE;
        __syncwarp();
    };
    if (planner) {
        if (lane == 0) {
            al.init();
            atomicAdd(A.queue + 1, 1), atomicAdd(A.queue + 3, 1);  // pairs running, started
            for (int b = 0; b < 3; ++b) S.at_end[b] = S.beyond[b] = S.retry[b] = 0;
            S.part.used = 0;
            if (A.free_slots == 0) S.beyond[0] = 1;  // trimmed from the first score on
        }
        __syncwarp();
        part_reset(S.part, lane);
        if (PIG || A.singletrack) {
            ring = alloc(PIG ? ring_arrays * rcap * 4 : (int64_t)R * 4 * ring_cap * 4);
            if (ring < 0) status = WFA_RETRY;
        }
        hdr_off = status == 0 ? alloc((int64_t)sizeof(ScoreHdr) * HDR_CHUNK) : -1;
        const int64_t d0 = hdr_off < 0 ? -1 : PIG ? ring : alloc(16);  // piggyback: M's slot 0
        if (status == 0 && d0 < 0) status = WFA_RETRY;
        if (status == 0) {
            // M[0] = {0} on diagonal 0, extended
            const int32_t o0 = (int32_t)lcp1(A, PR, pat, txt, 0, 0);
            if (lane == 0) {
                ctab[0] = hdr_off, *(int32_t *)(A.pool + d0) = o0;
                if (PIG) {
                    ((uint32_t *)(A.pool + d0))[rcap] = 0u;
                    ((uint32_t *)(A.pool + d0))[2 * rcap] = BT_NULL;  // the start (0, 0)
                }
            }
            __syncwarp();
            set_hdr(0, lane == 0 ? CompHdr{0, 0, 0, PIG ? rcap : 0, d0} : NUL);
            if (tlen - plen == 0 && o0 >= tlen) end_score = 0;
        }
        if (status != 0 || end_score == 0) {
            if (lane == 0) S.plan[0].op = WOP_DONE;
        } else {
            plan_next(S.plan[0]);
        }
    }
    __syncthreads();
    bool trimmed = false;
    int op = S.plan[0].op;
    for (int it = 0; op == WOP_COMPUTE; ++it) {
        const WidePlan &now = S.plan[it & 1];
        WidePlan &next = S.plan[(it + 1) & 1];
        if (!planner) {
            int told = 0;
            if constexpr (PIG) {
                int kmin[5], kmax[5];
                bool reached = false, past = false, ok = true;
#pragma unroll
                for (int c = 0; c < 5; ++c) kmin[c] = INT_MAX, kmax[c] = INT_MIN;
                // a warp whose first diagonal lies beyond the wavefront has none in the trip
                for (int kb = now.lo; kb + (tid & ~31) <= now.hi && ok; kb += NT * PIG_U)
                    ok = pig_trip(A, PR, pat, txt, kb, tid, NT, now.lo, now.hi, now.in, now.out, now.mask, now.out[CM].pad,
                                  al, bnext, bend, kmin, kmax, reached, past);
                if (trimmed) fold_partials(kmin, kmax, reached, S.part);
                if (!ok && lane == 0) S.retry[it % 3] = 1;
                told = (__any_sync(0xffffffffu, reached) ? 1 : 0) | (__any_sync(0xffffffffu, past) ? 2 : 0);
            } else {
                told = trimmed ? plan_compute<AW_WFA_CTA_U, NT, false>(PR, B, pat, txt, now, 0, 1, S.part)
                               : plan_compute<AW_WFA_CTA_U, NT, false, false>(PR, B, pat, txt, now, 0, 1, S.part);
            }
            if (lane == 0 && (told & 1)) S.at_end[it % 3] = 1;
            if (lane == 0 && (told & 2)) S.beyond[it % 3] = 1;
        } else {
            if (lane == 0) S.at_end[(it + 1) % 3] = 0, S.beyond[(it + 1) % 3] = 0, S.retry[(it + 1) % 3] = 0;
            if (!trimmed) commit(s, mine), plan_next(next);
        }
        __syncthreads();
        const bool stop = PIG && S.retry[it % 3] != 0, end = S.at_end[it % 3] != 0 && !stop;
        // (at the end too: the backtrace reads its header and those of the null scores before it)
        if (!stop && (trimmed || (!end && S.beyond[it % 3]))) {
            if (!trimmed) {
                // from here on the trimmed ends count, and the plan made meanwhile is dropped
                if (!planner) plan_trim(PR, now, tid, NT, S.part);
                else s = now.s, slot = s % R, num_null = 0, status = 0;
                trimmed = true;
                __syncthreads();
            }
            if (planner) {
                CompHdr out = lane < 5 ? now.out[lane] : NUL;
                if (lane < 5 && (now.mask >> lane & 1)) {
                    // no diagonal in the matrix: the empty range [lo, lo-1] of the scan
                    if (S.part.k[lane] == INT_MIN) out.hi = out.lo - 1;
                    else out.lo = -S.part.k[5 + lane], out.hi = S.part.k[lane];
                }
                __syncwarp();
                part_reset(S.part, lane);
                commit(now.s, out);
                if (!end) plan_next(next);
            }
            __syncthreads();
        }
        if (planner && end) end_score = now.s, status = 0;
        if (planner && stop) status = WFA_RETRY;
        op = end || stop ? WOP_DONE : next.op;
    }
    if (PIG && !planner && lane == 0) atomicAdd(&S.part.used, (unsigned long long)al.total());
    if (PIG) __syncthreads();
    if (planner && lane == 0) {
        if (!PIG) al.cur = cur;
        finish_pair<PIG>(A, PR, idx, pat, txt, ctab, HR, status, end_score, end_score >= 0 ? end_score : s,
                         al.total() + (PIG ? (int64_t)S.part.used : 0));
        atomicSub(A.queue + 1, 1);
        give_back(pool_of(A), al);
    }
    __syncthreads();
    if (PIG && !planner && lane == 0) give_back(pool_of(A), al);
}

// Build-time tuning of the warp kernel: CTAs per SM the registers are sized for (4 warps
// each), and diagonals per lane in flight in the high-memory compute step.
#ifndef AW_WFA_MINB
#define AW_WFA_MINB 4
#endif
#ifndef AW_WFA_WARP_U
#define AW_WFA_WARP_U 2
#endif
constexpr int WU = AW_WFA_WARP_U;

// Threads of a CTA: the long pairs' planning warp comes on top.
constexpr int wfa_threads(int nt) { return nt + 32; }

template <bool PIG, int NT>
__global__ void __launch_bounds__(wfa_threads(NT), NT > WFA_CTA ? 1 : PIG ? 3 : AW_WFA_MINB) wfa_kernel(WfaArgs A, RingShape rs) {
    const int lane = threadIdx.x & 31;
    const WfaPen P = A.pen;
    extern __shared__ CompHdr hring_all[];
    __shared__ Alloc allocs[wfa_threads(NT) / 32];
    Alloc &al = allocs[threadIdx.x >> 5];
    // the long pairs first, each on the whole CTA (the first warp's header ring serves the
    // planner; the warps take their own rings afterwards)
    __shared__ CtaShared S;
    for (;;) {
        if (threadIdx.x == 0) S.next = A.n_long > 0 ? atomicAdd(A.queue + A.q_long, 1) : A.n_long;
        __syncthreads();
        const int pi = S.next;
        __syncthreads();
        if (pi >= A.n_long) break;
        cta_open<PIG, NT>(A, A.order_long[pi], HdrRing{hring_all, rs}, S, PIG ? al : allocs[NT / 32]);
    }
    const HdrRing HR{hring_all + (threadIdx.x >> 5) * rs.entries(), rs};
    for (; A.n > 0;) {
        int pi = 0;
        if (lane == 0) pi = atomicAdd(A.queue, 1);
        pi = __shfl_sync(0xffffffffu, pi, 0);
        if (pi >= A.n) break;
        if (lane == 0) atomicAdd(A.queue + 1, 1), atomicAdd(A.queue + 3, 1);  // pairs running, started
        const int idx = A.order[pi];
        const WfaPairDev PR = A.pairs[idx];
        const int plen = PR.plen, tlen = PR.tlen;
        const uint8_t *pat = A.pat + PR.poff, *txt = A.txt + PR.toff;
        const Bases bases = bases_of(A, PR);
        int64_t *ctab = A.ctab + PR.ctab_off;
        if (lane == 0) al.init();
        uint32_t bnext = 0, bend = 0;  // this lane's reserved piggyback blocks
        int status = 0, end_score = -1;
        // piggyback rings, each slot three arrays (offsets, packed CIGARs, links) of rcap
        // elements: M keeps its last SR scores, I1/D1 their last e1+1 and I2/D2 their last
        // e2+1 (the only scores the compute step reads them from); grown by reallocation
        const int SR = A.max_score_scope, R1 = P.e1 + 1, R2 = P.e2 + 1;
        const int64_t ring_arrays = 3 * (int64_t)(SR + 2 * R1 + 2 * R2);
        int rcap = 0;
        int64_t rbase = -1;
        if constexpr (PIG) {
            rcap = 32;
            rbase = warp_alloc(A, al, ring_arrays * rcap * 4, lane);
            if (rbase < 0) status = WFA_RETRY;
        }
        // Singletrack ring for I/D: R slots x 4 components x cap offsets
        const int R = (P.e1 > P.e2 ? P.e1 : P.e2) + 1;
        const int ring_cap = plen + tlen + 8;
        int64_t ring = -1;
        if (A.singletrack) {
            ring = warp_alloc(A, al, (int64_t)R * 4 * ring_cap * 4, lane);
            if (ring < 0) status = WFA_RETRY;
        }
        // score 0
        int64_t h0 = -1;
        if (status == 0) {
            h0 = warp_alloc(A, al, (int64_t)sizeof(ScoreHdr) * HDR_CHUNK, lane);
            if (h0 < 0) status = WFA_RETRY;
        }
        int64_t d0 = -1;
        if (status == 0) {
            if constexpr (PIG) d0 = rbase;  // slot 0, component M
            else d0 = warp_alloc(A, al, 16, lane);
            if (d0 < 0) status = WFA_RETRY;
        }
        if (status == 0 && lane == 0) {
            ctab[0] = h0;
            ScoreHdr *H = (ScoreHdr *)(A.pool + h0);
            for (int c = 0; c < 5; ++c) H->c[c] = CompHdr{1, -1, 0, 0, 0};
            H->c[CM] = CompHdr{0, 0, 0, PIG ? rcap : 0, d0};
            *(int32_t *)(A.pool + d0) = 0;
            if constexpr (PIG) {
                ((uint32_t *)(A.pool + d0))[rcap] = 0u;
                ((uint32_t *)(A.pool + d0))[2 * rcap] = BT_NULL;  // the start (0, 0)
            }
            for (int c = 0; c < 5; ++c) HR.put(c, 0, H->c[c]);
        }
        __syncwarp();
        const int k_end = tlen - plen;
        int s = 0, num_null = 0;
        bool fused_reached = false;  // the compute step's extension reached the end (this lane)
        const int smax = PR.ctab_cap * HDR_CHUNK - 1;
        while (status == 0) {
            // ---- extend M[s] and check the end.  The compute step below extends M[s] as it
            // computes it (fused), so here only M[0] is extended.
            {
                const CompHdr m = HR.get(A, ctab, CM, s);
                bool reached = false;
                if (m.lo <= m.hi) {
                    if (s == 0) {
                        int32_t *d = (int32_t *)(A.pool + m.off);
                        for (int k0 = m.lo + lane; k0 <= m.hi; k0 += 128) {
                            int32_t o[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const int k = k0 + 32 * u;
                                o[u] = k <= m.hi ? d[k - m.base] : WF_NULL;
                            }
                            extend_n<4>(PR, bases_of(A, PR), pat, txt, k0, 32, o);
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const int k = k0 + 32 * u;
                                if (k <= m.hi && o[u] != WF_NULL) d[k - m.base] = o[u];
                                // end-to-end check on the lane that holds diagonal tlen-plen
                                if (k == k_end && o[u] != WF_NULL && o[u] >= tlen) reached = true;
                            }
                        }
                    } else {
                        reached = fused_reached;
                    }
                    if (__any_sync(0xffffffffu, reached)) {
                        end_score = s;
                        break;
                    }
                } else if (num_null > A.max_score_scope) {
                    status = -3;  // end unreachable (cannot happen end-to-end without heuristics)
                    break;
                }
            }
            // ---- compute s+1
            ++s;
            if (s > smax) {
                status = WFA_OVERFLOW;
                break;
            }
            if (s % HDR_CHUNK == 0) {
                const int64_t hb = warp_alloc(A, al, (int64_t)sizeof(ScoreHdr) * HDR_CHUNK, lane);
                if (hb < 0) {
                    status = WFA_RETRY;
                    break;
                }
                if (lane == 0) ctab[s / HDR_CHUNK] = hb;
                __syncwarp();
            }
            ScoreHdr *OH = hdr_ptr(A, ctab, s);
            const CompHdr NUL{1, -1, 0, 0, 0};
            const int sm = s - P.x, so1 = s - P.o1 - P.e1, se1 = s - P.e1, so2 = s - P.o2 - P.e2, se2 = s - P.e2;
            const CompHdr m_misms = sm >= 0 ? HR.get(A, ctab, CM, sm) : NUL;
            const CompHdr m_open1 = so1 >= 0 ? HR.get(A, ctab, CM, so1) : NUL;
            const CompHdr i1 = se1 >= 0 ? HR.get(A, ctab, CI1, se1) : NUL;
            const CompHdr d1 = se1 >= 0 ? HR.get(A, ctab, CD1, se1) : NUL;
            const CompHdr m_open2 = so2 >= 0 ? HR.get(A, ctab, CM, so2) : NUL;
            const CompHdr i2 = se2 >= 0 ? HR.get(A, ctab, CI2, se2) : NUL;
            const CompHdr d2 = se2 >= 0 ? HR.get(A, ctab, CD2, se2) : NUL;
            const bool n_mm = m_misms.lo > m_misms.hi, n_o1 = m_open1.lo > m_open1.hi, n_i1 = i1.lo > i1.hi,
                       n_d1 = d1.lo > d1.hi, n_o2 = m_open2.lo > m_open2.hi, n_i2 = i2.lo > i2.hi,
                       n_d2 = d2.lo > d2.hi;
            if (n_mm && n_o1 && n_i1 && n_d1 && n_o2 && n_i2 && n_d2) {
                if (lane == 0)
                    for (int c = 0; c < 5; ++c) OH->c[c] = NUL, HR.put(c, s, NUL);
                __syncwarp();
                ++num_null;
                fused_reached = false;
                continue;
            }
            num_null = 0;
            fused_reached = false;
            // limits (null inputs contribute lo=1, hi=-1)
            int lo = m_misms.lo, hi = m_misms.hi;
            lo = min(lo, m_open1.lo - 1), hi = max(hi, m_open1.hi + 1);
            lo = min(lo, i1.lo + 1), hi = max(hi, i1.hi + 1);
            lo = min(lo, d1.lo - 1), hi = max(hi, d1.hi - 1);
            lo = min(lo, m_open2.lo - 1), hi = max(hi, m_open2.hi + 1);
            lo = min(lo, i2.lo + 1), hi = max(hi, i2.hi + 1);
            lo = min(lo, d2.lo - 1), hi = max(hi, d2.hi - 1);
            const bool a_i1 = !n_o1 || !n_i1, a_d1 = !n_o1 || !n_d1, a_i2 = !n_o2 || !n_i2, a_d2 = !n_o2 || !n_d2;
            const int width = hi - lo + 1;
            // a wavefront wider than a warp's share: the cluster kernel re-runs the pair.  Above
            // wide_width always; above wide_width_tail once every pair has started and at most
            // wide_tail_pairs still run on warps (the batch's tail, whose idle SMs the cluster
            // kernel puts to work)
            if (!PIG && A.wide_width > 0 && width > A.wide_width_tail) {
                int drained = 0;
                if (lane == 0)
                    drained = *(volatile int32_t *)(A.queue + 3) >= A.n_all &&
                              *(volatile int32_t *)(A.queue + 1) <= A.wide_tail_pairs;
                drained = __shfl_sync(0xffffffffu, drained, 0);
                if (width > A.wide_width || drained) {
                    status = WFA_WIDE;
                    break;
                }
            }
            CompHdr out[5];
            for (int c = 0; c < 5; ++c) out[c] = NUL;
            const bool alloc_c[5] = {true, a_i1, a_d1, a_i2, a_d2};
            if constexpr (PIG) {
                if (width > rcap) {
                    const int nc = max(2 * rcap, (width + 3) & ~3);
                    const int64_t nb = warp_alloc(A, al, ring_arrays * nc * 4, lane);
                    if (nb < 0) {
                        status = WFA_RETRY;
                        break;
                    }
                    rcap = nc, rbase = nb;
                }
                for (int c = 0; c < 5; ++c)
                    if (alloc_c[c])
                        out[c] = CompHdr{lo, hi, lo, rcap, rbase + pig_slot(c, s, SR, R1, R2) * rcap * 4};
            } else {
                const int64_t wb = (((int64_t)width * 4) + 15) & ~(int64_t)15;
                int nstore = 1;
                if (!A.singletrack) nstore += (int)a_i1 + (int)a_d1 + (int)a_i2 + (int)a_d2;
                if (A.singletrack && width > ring_cap) {
                    status = WFA_OVERFLOW;
                    break;
                }
                const int64_t blk = warp_alloc(A, al, wb * nstore, lane);
                if (blk < 0) {
                    status = WFA_RETRY;
                    break;
                }
                int64_t o = blk;
                for (int c = 0; c < 5; ++c) {
                    if (!alloc_c[c]) continue;
                    int64_t place;
                    if (c == CM || !A.singletrack) place = o, o += wb;
                    else place = ring + ((int64_t)((s % R) * 4 + (c - 1)) * ring_cap) * 4;
                    out[c] = CompHdr{lo, hi, lo, 0, place};
                }
            }
            // trimmed ends (wavefront/wavefront_compute.c:654-690): the lowest and highest
            // diagonal whose offset lies in the matrix, per component, from the lanes' values
            int kmin[5], kmax[5];
#pragma unroll
            for (int c = 0; c < 5; ++c) kmin[c] = INT_MAX, kmax[c] = INT_MIN;
            if constexpr (PIG) {
                // PIG_U diagonals per lane at a time (every lane runs every trip: the block
                // reservation is warp-wide)
                const CompHdr in7[7] = {m_misms, m_open1, i1, d1, m_open2, i2, d2};
                int mask = 0;
                for (int c = 0; c < 5; ++c) mask |= alloc_c[c] ? 1 << c : 0;
                for (int kb = lo; kb <= hi; kb += 32 * PIG_U) {
                    bool beyond;  // not used
                    if (!pig_trip(A, PR, pat, txt, kb, lane, 32, lo, hi, in7, out, mask, rcap, al, bnext, bend, kmin, kmax,
                                  fused_reached, beyond)) {
                        status = WFA_RETRY;
                        break;
                    }
                }
                if (status != 0) break;
            } else {
                const InHdr h[7] = {in_hdr(A, m_misms), in_hdr(A, m_open1), in_hdr(A, i1), in_hdr(A, d1),
                                    in_hdr(A, m_open2), in_hdr(A, i2),      in_hdr(A, d2)};
                int32_t *dst[5];
                int ilo = INT_MIN, ihi = INT_MAX;  // the diagonals that every input has
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    dst[c] = alloc_c[c] ? (int32_t *)(A.pool + out[c].off) : nullptr;
                    if (!alloc_c[c]) ihi = INT_MIN;
                }
#pragma unroll
                for (int j = 0; j < 7; ++j) ilo = max(ilo, h[j].lo), ihi = min(ihi, h[j].hi);
                bool beyond;  // not used
                for (int kw = lo; kw <= hi; kw += 32 * WU) {
                    if (kw > ilo && kw + 32 * WU <= ihi)
                        wf_trip<WU, 32, true, false, true, false>(PR, bases, pat, txt, h, dst, lo, hi, kw + lane, kmin,
                                                                  kmax, fused_reached, beyond);
                    else if (hi - kw >= 32)
                        wf_trip<WU, 32, false, true, true, false>(PR, bases, pat, txt, h, dst, lo, hi, kw + lane, kmin,
                                                                  kmax, fused_reached, beyond);
                    else
                        wf_trip<1, 32, false, true, true, false>(PR, bases, pat, txt, h, dst, lo, hi, kw + lane, kmin,
                                                                 kmax, fused_reached, beyond);
                }
            }
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                if (!alloc_c[c]) continue;
                const int th = __reduce_max_sync(0xffffffffu, kmax[c]);
                const int tl = __reduce_min_sync(0xffffffffu, kmin[c]);
                // no diagonal in the matrix: the empty range [lo, lo-1] of the scan
                if (th == INT_MIN) out[c].hi = out[c].lo - 1;
                else out[c].lo = tl, out[c].hi = th;
            }
            if (lane == 0)
                for (int c = 0; c < 5; ++c) OH->c[c] = out[c], HR.put(c, s, out[c]);
            __syncwarp();
        }
        // ---- backtrace (lane 0)
        if (lane == 0) {
            finish_pair<PIG>(A, PR, idx, pat, txt, ctab, HR, status, end_score, s, al.total());
            atomicSub(A.queue + 1, 1);
        }
        __syncwarp();
        if (lane == 0) give_back(pool_of(A), al);
    }
}

// ---------------------------------------------------------------------------------------
// Cluster kernel for pairs whose wavefronts outgrow a warp (high memory: standard and
// Singletrack).  One cluster of CL CTAs per pair; in each, WIDE_CW warps compute and one plans.
// A pair is a chain of scores, each as long as one pass over the wavefront and a barrier of the
// cluster take, so nothing else may stand in it.
//
// Trimming a wavefront to the diagonals inside the matrix needs the ends of all CTAs.  But the
// cells that it cuts off are null, which reads the same stored or not, or offsets beyond the end
// of a sequence; until there is one of those, the ranges depend on nothing but the score (they come
// out a few diagonals wider than trimmed ones), and the planners go ahead of the warps:
//   1. the computing warps of all CTAs compute and extend the diagonals of the planned score
//      (plan_open);
//   2. meanwhile the planning warps plan the next one, a lane per input and per component.
//      Every planner holds the same state (the headers of the last scores in shared-memory
//      rings, the pool position), so all plans agree without being exchanged;
//   3. cluster barrier.
// A warp that computes an offset beyond the end says so in every CTA's shared memory before the
// barrier, and from that score on wavefronts are trimmed: its own is, from what is stored, and
// the next score is planned again; after that the warps fold their trimmed ends into their CTA's
// partials (plan_compute), and after the barrier the planners gather all CTAs' partials through
// distributed shared memory, finish the score's headers and plan the next one.  The end is
// announced in the same way.
// Measured on one pair at 12% in us per score, with trimmed ends gathered and the next score planned
// by the first warp after each barrier, and now: 10 kb 5.4 -> 2.8, 24 kb 7.7 -> 3.5.
//
// Pool space is carved deterministically out of reserve chunks that the first CTA's planner
// (the leader) takes from the pool one score ahead of need and announces to every CTA
// through distributed shared memory before the barrier; the first CTA's planner alone writes the
// pool copy of the headers and the chunk table that the backtrace reads.  The cell arithmetic and
// the backtrace are the warp kernel's, so the results are identical.  Offsets written by other
// CTAs are ordered by the barrier's release/acquire.
constexpr int WIDE_SEQ_WORDS = 12 * 1024;  // 2-bit words of a pair kept in shared memory
constexpr int WIDE_CW = 12, WIDE_NT = 32 * (WIDE_CW + 1);
constexpr int WIDE_MAX_CL = 16;  // CTAs of a cluster, at most
constexpr int WIDE_CHUNKS = 8;  // reserve chunks a planner keeps track of (a ring)

// A reserve chunk announced by the leader: for pair `tag`, the planners' chunk number `seq`
// (off < 0: the pool is exhausted).
struct WideAnn {
    int tag, seq;
    int64_t off, len;
};

// The planner's state (the same in all lanes of every CTA's planning warp).
struct WidePlanner {
    int pi, idx;  // queue position and pair
    int s, num_null, status, end_score, smax, R, ring_cap;
    int lo_all, hi_all;  // the union of the planned diagonal ranges so far
    int64_t ring, hdr_off, ctab_off;
    int s_hdr, committed;  // the first score of the header chunk hdr_off, the last score with headers
    int plen, tlen;
    int slot;            // s mod R
    int64_t cur, end;    // carving position in the current chunk
    int64_t used;        // bytes carved
    int nchunks, cidx;   // chunks received, chunk being carved
    bool exhausted;
};

// Reserve chunk size: large (few pool atomics), smaller in a small pool.
__device__ __forceinline__ int64_t wide_chunk(const WfaArgs &A, int64_t need) {
    const int64_t base = min((int64_t)64 << 20, max((int64_t)1 << 20, A.pool_bytes / 64));
    return ((max(base, 2 * need) + 255) & ~(int64_t)255);
}

__global__ void __launch_bounds__(WIDE_NT, 1) wfa_wide_kernel(WfaArgs A, RingShape rs) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int CL = (int)cl.num_blocks();
    const int rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31;
    const bool planner = tid >= 32 * WIDE_CW;
    const bool leader = rank == 0 && planner && lane == 0;
    const WfaPen P = A.pen;
    // plan of step it in plan[it & 1], its partials in part[it & 1] (part[2]: of the first trimmed
    // score), its end and beyond flags at it % 3 (cleared at step it + 2)
    __shared__ WidePlan plan[2];
    __shared__ WidePart part[3];
    __shared__ int at_end[3], beyond[3];
    __shared__ WideAnn ann[2];     // reserve chunks announced before the barrier of step it (it & 1)
    __shared__ WideAnn pstart[2];  // the pair of the np-th pair start (np & 1): tag = queue position,
                                   // seq = pair, off/len = its first chunk
    __shared__ int64_t qoff[WIDE_CHUNKS], qlen[WIDE_CHUNKS];  // the planner's chunks
    // the header ring, then the pair's packed sequences if they fit (the barrier of a score drops
    // the L1 lines, so that from global memory the extension would wait for the L2 each time)
    extern __shared__ CompHdr wring[];
    const HdrRing HR{wring, rs};
    uint64_t *const seqs = (uint64_t *)(wring + rs.entries());
    const PlanLane L = plan_lane(P, lane);
    // where this lane of a planner reads its input and writes its component
    const CompHdr *const rd = HR.at(L.comp, 0);
    CompHdr *const wr = HR.at(min(lane, 4), 0);
    const int rd_mask = HR.mask(L.comp), wr_mask = HR.mask(min(lane, 4));
    if (planner && lane < 2) ann[lane] = WideAnn{-1, -1, -1, 0};
    const CompHdr NUL{1, -1, 0, 0, 0};
    WidePlanner W{};
    CompHdr mine = NUL;  // a planner's lane c < 5: component c's header of the planned score
    int it = 0, np = 0;
    // every CTA of the cluster has started (and cleared ann) before one writes another's shared memory
    cl.sync();

    // ---- planner helpers (all lanes of the planning warp)
    auto carve = [&](int64_t bytes) -> int64_t {
        bytes = (bytes + 15) & ~(int64_t)15;
        while (W.cur + bytes > W.end) {
            if (W.cidx + 1 >= W.nchunks) return -1;
            ++W.cidx;
            W.cur = qoff[W.cidx % WIDE_CHUNKS];
            W.end = W.cur + qlen[W.cidx % WIDE_CHUNKS];
            if (W.cur < 0) return -1;
        }
        const int64_t r = W.cur;
        W.cur += bytes, W.used += bytes;
        return r;
    };
    // bytes the next plan may carve: one header chunk and the stored components over the
    // planned range widened by one diagonal per side
    auto need_next = [&]() -> int64_t {
        const int64_t w = (int64_t)(W.hi_all - W.lo_all) + 3;
        return (int64_t)sizeof(ScoreHdr) * HDR_CHUNK + (A.singletrack ? 1 : 5) * (w * 4 + 16) + 64;
    };
    // the next plan's carves fit: in the current chunk's tail, or in one queued chunk (a
    // carve that does not fit moves on to the next chunk)
    auto reserve_ok = [&]() -> bool {
        const int64_t need = need_next();
        bool ok = W.end - W.cur >= need;
        if (ok) return true;
        for (int j = W.cidx + 1; j < W.nchunks; ++j) ok |= qlen[j % WIDE_CHUNKS] >= need;
        return ok;
    };
    // lane c < 5: component c's header of score sc (the first CTA's planner writes the pool copy)
    auto set_hdr = [&](int sc, const CompHdr &o) {
        if (lane < 5) {
            if (rank == 0) {
                const int64_t off = sc >= W.s_hdr ? W.hdr_off : A.ctab[W.ctab_off + sc / HDR_CHUNK];
                ((ScoreHdr *)(A.pool + off))[sc % HDR_CHUNK].c[lane] = o;
            }
            wr[sc & wr_mask] = o;
        }
        __syncwarp();
    };
    // the headers of score sc, and of the null scores before it
    auto commit = [&](int sc, const CompHdr &o) {
        for (int z = W.committed + 1; z < sc; ++z) set_hdr(z, NUL);
        set_hdr(sc, o);
        W.committed = sc;
    };
    // a reserve chunk announced at step k
    auto take_ann = [&](int k) {
        const WideAnn &a = ann[k & 1];
        if (a.tag == W.pi && a.seq == W.nchunks) {
            if (lane == 0) qoff[W.nchunks % WIDE_CHUNKS] = a.off, qlen[W.nchunks % WIDE_CHUNKS] = a.len;
            __syncwarp();
            ++W.nchunks;
            if (a.off < 0) W.exhausted = true;
        }
    };
    // the headers of plan q's score with the trimmed ends of all CTAs (partials b)
    auto finish_score = [&](const WidePlan &q, int b) {
        // lane i < 10: value i of every CTA's partials
        int v = INT_MIN;
        if (lane < 10) {
#pragma unroll
            for (int r = 0; r < WIDE_MAX_CL; ++r)
                if (r < CL) v = max(v, *cl.map_shared_rank(&part[b].k[lane], r));
        }
        const int top = v, bottom = __shfl_down_sync(0xffffffffu, v, 5);
        CompHdr out = lane < 5 ? q.out[lane] : NUL;
        if (lane < 5 && (q.mask >> lane & 1)) {
            // no diagonal in the matrix: the empty range [lo, lo-1] of the scan
            if (top == INT_MIN) out.hi = out.lo - 1;
            else out.lo = -bottom, out.hi = top;
        }
        commit(q.s, out);
    };
    // plans the next score with a non-null input into `q`; op = DONE with W.status set if the
    // pair stops
    auto plan_next = [&](WidePlan &q) {
        for (;;) {
            ++W.s;
            W.slot = W.slot + 1 == W.R ? 0 : W.slot + 1;
            const int s = W.s;
            if (s > W.smax) {
                W.status = WFA_OVERFLOW;
                break;
            }
            if (s % HDR_CHUNK == 0) {
                const int64_t hb = carve((int64_t)sizeof(ScoreHdr) * HDR_CHUNK);
                if (hb < 0) {
                    W.status = WFA_RETRY;
                    break;
                }
                W.hdr_off = hb, W.s_hdr = s;
                if (leader) A.ctab[W.ctab_off + s / HDR_CHUNK] = hb;
                __syncwarp();
            }
            // the scores since the last committed one are null
            CompHdr in = NUL;
            if (lane < 7 && s - L.dist >= 0 && s - L.dist <= W.committed) in = rd[(s - L.dist) & rd_mask];
            const unsigned some = __ballot_sync(0xffffffffu, lane < 7 && in.lo <= in.hi);
            if (!some) {
                // the top of the next step: M[s] is empty
                if (++W.num_null > A.max_score_scope) {
                    W.status = -3;
                    break;
                }
                continue;
            }
            W.num_null = 0;
            int lo, hi, mask;
            plan_limits(L, lane, in, some, lo, hi, mask);
            // no diagonal beyond these has a cell
            lo = max(lo, -W.plen), hi = min(hi, W.tlen);
            W.lo_all = min(W.lo_all, lo), W.hi_all = max(W.hi_all, hi);
            const int width = hi - lo + 1;
            const int64_t wb = (((int64_t)width * 4) + 15) & ~(int64_t)15;
            if (A.singletrack && width > W.ring_cap) {
                W.status = WFA_OVERFLOW;
                break;
            }
            const int64_t blk = carve(wb * (A.singletrack ? 1 : __popc(mask)));
            if (blk < 0) {
                W.status = WFA_RETRY;
                break;
            }
            if (lane < 5) {
                CompHdr out = NUL;
                if (mask >> lane & 1)
                    out = CompHdr{lo, hi, lo, 0,
                                  lane == CM || !A.singletrack ? blk + wb * __popc(mask & ((1 << lane) - 1))
                                                               : W.ring + ((int64_t)(W.slot * 4 + (lane - 1)) * W.ring_cap) * 4};
                mine = out;
                q.out[lane] = out;
                q.dst[lane] = mask >> lane & 1 ? (int32_t *)(A.pool + out.off) : nullptr;
            }
            if (lane < 7) q.view[lane] = in_hdr(A, in);
            plan_inner(q, mask, lane, in);
            if (lane == 0) q.op = WOP_COMPUTE, q.lo = lo, q.hi = hi, q.mask = mask, q.s = s;
            __syncwarp();
            return;
        }
        if (lane == 0) q.op = WOP_DONE;
        __syncwarp();
    };
    // the leader reserves the next plan's space ahead of need
    auto reserve = [&](int k) {
        if (leader && !W.exhausted && W.nchunks - W.cidx < WIDE_CHUNKS - 1 && !reserve_ok()) {
            int64_t len = wide_chunk(A, need_next());
            const int64_t off = pool_grab_rest(pool_of(A), len, need_next());
            const WideAnn a{W.pi, W.nchunks, off, off >= 0 ? len : 0};
            for (int c = 0; c < CL; ++c) *cl.map_shared_rank(&ann[k & 1], c) = a;
        }
        __syncwarp();
    };

    for (;;) {
        // ---- pair start: the leader takes the next pair and its first chunk
        if (leader) {
            WideAnn a{A.n, -1, -1, 0};
            const int pi = atomicAdd(A.queue, 1);
            if (pi < A.n) {
                const int idx = A.order[pi];
                const WfaPairDev PR = A.pairs[idx];
                const int R = (P.e1 > P.e2 ? P.e1 : P.e2) + 1;
                const int64_t ring_b = A.singletrack ? (int64_t)R * 4 * (PR.plen + PR.tlen + 8) * 4 + 16 : 0;
                const int64_t len = wide_chunk(A, ring_b + (int64_t)sizeof(ScoreHdr) * HDR_CHUNK + 4096);
                a = WideAnn{pi, idx, pool_grab(pool_of(A), len), len};
            }
            for (int c = 0; c < CL; ++c) *cl.map_shared_rank(&pstart[np & 1], c) = a;
        }
        cl.sync();
        it = 0;
        if (planner) {
            for (int b = 0; b < 3; ++b) part_reset(part[b], lane);
            if (lane < 3) at_end[lane] = 0, beyond[lane] = 0;
            const WideAnn a = pstart[np & 1];
            if (a.tag >= A.n) {
                if (lane == 0) plan[0].op = WOP_EXIT;
            } else {
                const WfaPairDev PR = A.pairs[a.seq];
                W = WidePlanner{};
                W.pi = a.tag, W.idx = a.seq, W.ctab_off = PR.ctab_off;
                W.smax = PR.ctab_cap * HDR_CHUNK - 1;
                W.R = (P.e1 > P.e2 ? P.e1 : P.e2) + 1;
                W.ring_cap = PR.plen + PR.tlen + 8;
                W.plen = PR.plen, W.tlen = PR.tlen;
                W.end_score = -1, W.lo_all = 0, W.hi_all = 0;
                W.ring = -1;
                if (lane == 0) qoff[0] = a.off, qlen[0] = a.len;
                __syncwarp();
                W.nchunks = 1, W.cidx = 0, W.cur = a.off, W.end = a.off + a.len;
                W.exhausted = a.off < 0;
                if (a.off < 0) W.status = WFA_RETRY;
                if (W.status == 0 && A.singletrack) {
                    W.ring = carve((int64_t)W.R * 4 * W.ring_cap * 4);
                    if (W.ring < 0) W.status = WFA_RETRY;
                }
                const int64_t h0 = W.status == 0 ? carve((int64_t)sizeof(ScoreHdr) * HDR_CHUNK) : -1;
                const int64_t d0 = h0 >= 0 ? carve(16) : -1;
                if (W.status == 0 && d0 < 0) W.status = WFA_RETRY;
                if (W.status == 0) {
                    // M[0] = {0} on diagonal 0, extended (every planner writes the same value)
                    const int32_t o0 = (int32_t)lcp1(A, PR, A.pat + PR.poff, A.txt + PR.toff, 0, 0);
                    W.hdr_off = h0;
                    if (leader) A.ctab[PR.ctab_off] = h0;
                    if (lane == 0) *(int32_t *)(A.pool + d0) = o0;
                    __syncwarp();
                    set_hdr(0, lane == 0 ? CompHdr{0, 0, 0, 0, d0} : NUL);
                    if (PR.tlen - PR.plen == 0 && o0 >= PR.tlen) W.end_score = 0;
                }
                if (W.status != 0 || W.end_score == 0) {
                    if (lane == 0) plan[0].op = WOP_DONE;
                } else {
                    plan_next(plan[0]);
                    reserve(1);  // announced in ann[1], read at step 0's planning
                }
            }
        }
        // flags and partials are clear in every CTA before another one's first step
        cl.sync();
        ++np;
        int op = plan[0].op;
        if (op == WOP_EXIT) break;
        const int pidx = pstart[(np - 1) & 1].seq;
        const WfaPairDev PR = A.pairs[pidx];
        const uint8_t *pat = A.pat + PR.poff, *txt = A.txt + PR.toff;
        Bases B = bases_of(A, PR);
        const int pw = (B.po + PR.plen) / 32 + 2, tw = (B.to + PR.tlen) / 32 + 2;
        const bool staged = PR.packed && op == WOP_COMPUTE && pw + tw <= WIDE_SEQ_WORDS;
        if (staged) {
            for (int i = tid; i < pw; i += WIDE_NT) seqs[i] = __ldg(B.p + i);
            for (int i = tid; i < tw; i += WIDE_NT) seqs[pw + i] = __ldg(B.t + i);
            B.p = seqs, B.t = seqs + pw;
            __syncthreads();
        }
        bool trimmed = false;
        while (op == WOP_COMPUTE) {
            const WidePlan &now = plan[it & 1];
            if (!planner) {
                // ---- 1. this warp's diagonals of the planned score
                int told;
                if (trimmed) told = plan_compute<2, 32 * WIDE_CW, false>(PR, bases_of(A, PR), pat, txt, now, rank, CL, part[it & 1]);
                else if (staged) told = plan_open<32 * (WIDE_CW - 1), true>(PR, B, pat, txt, now, rank, CL);
                else told = plan_open<32 * (WIDE_CW - 1), false>(PR, B, pat, txt, now, rank, CL);
                if (told && lane < CL) {
                    if (told & 1) *cl.map_shared_rank(&at_end[it % 3], lane) = 1;
                    if (told & 2) *cl.map_shared_rank(&beyond[it % 3], lane) = 1;
                }
            } else {
                // ---- 2. its headers, and the plan of the next one
                if (lane == 0) at_end[(it + 1) % 3] = 0, beyond[(it + 1) % 3] = 0;
                if (!trimmed) {
                    take_ann(it - 1);
                    commit(W.s, mine);
                    plan_next(plan[(it + 1) & 1]);
                }
                reserve(it);
            }
            // ---- 3.
            cl.sync();
            const bool end = at_end[it % 3] != 0;
            // (at the end too: the backtrace reads the headers of the null scores before it)
            if (trimmed || (!end && beyond[it % 3])) {
                if (!trimmed) {
                    if (!planner) plan_trim(PR, now, rank * 32 * WIDE_CW + tid, CL * 32 * WIDE_CW, part[2]);
                    cl.sync();
                }
                if (planner) {
                    if (trimmed) part_reset(part[(it + 1) & 1], lane);
                    else W.s = now.s, W.slot = now.s % W.R, W.num_null = 0, W.status = 0;  // drop the plan made meanwhile
                    take_ann(it);
                    finish_score(now, trimmed ? it & 1 : 2);
                    if (!end) plan_next(plan[(it + 1) & 1]);
                }
                trimmed = true;
                __syncthreads();
            }
            if (planner && end) W.end_score = now.s, W.status = 0;
            ++it;
            op = end ? WOP_DONE : plan[it & 1].op;
        }
        // ---- backtrace (leader)
        if (leader)
            finish_pair<false>(A, PR, W.idx, pat, txt, A.ctab + PR.ctab_off, HR, W.status, W.end_score, W.end_score >= 0 ? W.end_score : W.s,
                               W.used);
        cl.sync();
    }
}

}  // namespace

// Header rings for a penalty set: powers of two above each component's reach; no rings (pool
// reads) when they would take more than `cap` bytes.
static RingShape ring_shape(const WfaPen &P, int scope, int cap) {
    auto mask = [](int reach) {
        int n = 2;
        while (n <= reach && n < (1 << 20)) n <<= 1;
        return n - 1;
    };
    const RingShape r{mask(scope), mask(P.e1), mask(P.e2)};
    if ((int64_t)r.entries() * (int64_t)sizeof(CompHdr) > cap) return RingShape{-1, 0, 0};
    return r;
}
constexpr int WARP_RING_BYTES = 8 * 1024, WIDE_RING_BYTES = 96 * 1024;

template <bool PIG, int NT>
static cudaError_t launch_wfa_t(const WfaArgs &a, int ctas, cudaStream_t st) {
    const RingShape rs = ring_shape(a.pen, a.max_score_scope, WARP_RING_BYTES);
    const size_t smem = (size_t)(wfa_threads(NT) / 32) * rs.entries() * sizeof(CompHdr);
    if (smem > 48 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(wfa_kernel<PIG, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    wfa_kernel<PIG, NT><<<ctas, wfa_threads(NT), smem, st>>>(a, rs);
    return cudaGetLastError();
}

cudaError_t launch_wfa(const WfaArgs &a, int threads, int ctas, cudaStream_t st) {
    if (threads == WFA_BIG_CTA)
        return a.piggyback ? launch_wfa_t<true, WFA_BIG_CTA>(a, ctas, st) : launch_wfa_t<false, WFA_BIG_CTA>(a, ctas, st);
    return a.piggyback ? launch_wfa_t<true, WFA_CTA>(a, ctas, st) : launch_wfa_t<false, WFA_CTA>(a, ctas, st);
}

static cudaLaunchConfig_t wide_config(int ctas, int cl, size_t smem, cudaStream_t st, cudaLaunchAttribute *at) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(WIDE_NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// Dynamic shared memory of the cluster kernel, and what its launches need set; an
// error if the header ring of this score scope does not fit.
static cudaError_t wide_setup(const WfaPen &pen, int scope, int cl, RingShape &rs, size_t &smem) {
    rs = ring_shape(pen, scope, WIDE_RING_BYTES);
    if (rs.mm < 0 || cl > WIDE_MAX_CL) return cudaErrorInvalidValue;
    smem = (size_t)rs.entries() * sizeof(CompHdr) + WIDE_SEQ_WORDS * sizeof(uint64_t);
    cudaError_t e = cudaFuncSetAttribute(wfa_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && cl > 8) e = cudaFuncSetAttribute(wfa_wide_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

cudaError_t launch_wfa_wide(const WfaArgs &a, int clusters, int cl, cudaStream_t st) {
    RingShape rs;
    size_t smem;
    cudaError_t e = wide_setup(a.pen, a.max_score_scope, cl, rs, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = wide_config(clusters * cl, cl, smem, st, at);
    e = cudaLaunchKernelEx(&cfg, wfa_wide_kernel, a, rs);
    return e != cudaSuccess ? e : cudaGetLastError();
}

int wfa_wide_clusters(int cl, const WfaPen &pen, int scope) {
    RingShape rs;
    size_t smem;
    if (wide_setup(pen, scope, cl, rs, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = wide_config(cl, cl, smem, 0, at);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, (void *)wfa_wide_kernel, &cfg) == cudaSuccess) return n;
    cudaGetLastError();
    return 0;
}

namespace {

__device__ __forceinline__ uint64_t code2(uint8_t c) {
    return c == 'C' ? 1u : c == 'G' ? 2u : c == 'T' ? 3u : 0u;
}

// One thread per word of 32 bases.
__global__ void wfa_pack_kernel(const uint8_t *src, int64_t nbytes, uint64_t *dst, int64_t nwords) {
    const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nwords) return;
    uint64_t r = 0;
    const int64_t b0 = w * 32;
    if (b0 + 32 <= nbytes) {
        const uint4 a = *reinterpret_cast<const uint4 *>(src + b0), b = *reinterpret_cast<const uint4 *>(src + b0 + 16);
        const uint32_t wd[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 32; ++i) r |= code2((uint8_t)(wd[i >> 2] >> (8 * (i & 3)))) << (2 * i);
    } else {
        for (int i = 0; i < 32 && b0 + i < nbytes; ++i) r |= code2(src[b0 + i]) << (2 * i);
    }
    dst[w] = r;
}

// One warp per pair: packed = no byte other than A, C, G, T in the pattern and the text.
__global__ void wfa_classify_kernel(const uint8_t *pat, const uint8_t *txt, WfaPairDev *pairs, int n) {
    const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= n) return;
    const WfaPairDev P = pairs[i];
    bool bad = false;
    for (int j = lane; j < P.plen && !bad; j += 32) {
        const uint8_t c = pat[P.poff + j];
        bad = !(c == 'A' || c == 'C' || c == 'G' || c == 'T');
    }
    for (int j = lane; j < P.tlen && !bad; j += 32) {
        const uint8_t c = txt[P.toff + j];
        bad = !(c == 'A' || c == 'C' || c == 'G' || c == 'T');
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) pairs[i].packed = bad ? 0 : 1;
}

}  // namespace

cudaError_t launch_wfa_pack(const uint8_t *pat, int64_t pbytes, uint64_t *ppat, const uint8_t *txt, int64_t tbytes,
                            uint64_t *ptxt, WfaPairDev *pairs, int n, cudaStream_t st) {
    const int64_t pw = (pbytes + 31) / 32 + 2, tw = (tbytes + 31) / 32 + 2;
    wfa_pack_kernel<<<(unsigned)((pw + 255) / 256), 256, 0, st>>>(pat, pbytes, ppat, pw);
    wfa_pack_kernel<<<(unsigned)((tw + 255) / 256), 256, 0, st>>>(txt, tbytes, ptxt, tw);
    if (n > 0) wfa_classify_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(pat, txt, pairs, n);
    return cudaGetLastError();
}

int wfa_occupancy(bool piggyback, int threads, const WfaPen &pen, int scope) {
    const int nt = wfa_threads(threads);
    const size_t smem = (size_t)(nt / 32) * ring_shape(pen, scope, WARP_RING_BYTES).entries() * sizeof(CompHdr);
    const void *k = threads == WFA_BIG_CTA
                        ? (piggyback ? (const void *)wfa_kernel<true, WFA_BIG_CTA> : (const void *)wfa_kernel<false, WFA_BIG_CTA>)
                        : (piggyback ? (const void *)wfa_kernel<true, WFA_CTA> : (const void *)wfa_kernel<false, WFA_CTA>);
    if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int nb = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, nt, smem);
    return e == cudaSuccess ? nb : 1;
}

}  // namespace aw
