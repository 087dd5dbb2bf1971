// Internal types of the WFA kernel (wfa.cu) and its host layer (wfa_api.cu).
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

namespace aw {

// WF status codes (WFA2-lib wavefront/wfa.h:46-55) plus internal retry/overflow.
constexpr int WFA_COMPLETED = 0;
constexpr int WFA_OOM = -200;
constexpr int WFA_UNATTAINABLE = -300;
constexpr int WFA_RETRY = -1000;     // device pool exhausted: re-run in a later round
constexpr int WFA_OVERFLOW = -1001;  // a per-pair bound was exceeded
constexpr int WFA_WIDE = -1002;      // wavefront wider than a warp's share: re-run by the cluster kernel

struct WfaPen {
    int x, o1, e1, o2, e2;
};

struct WfaPairDev {
    int64_t poff, toff;    // padded pattern / text in the sequence arenas (8-byte aligned)
    int32_t plen, tlen;
    int64_t ops_off;       // CIGAR operation slot (plen + tlen + 8 chars)
    int64_t ctab_off;      // header-chunk table (int64 pool offsets), ctab_cap entries
    int32_t ctab_cap;
    int32_t packed;        // 1: pattern and text are uppercase ACGT only (set on the device)
};

struct WfaOutDev {
    int32_t status, score, n_ops, final_s;
    int64_t mem_bytes;
};

// Counters of the wavefront pool, zero at the start of a round.
struct WfaPoolCtl {
    unsigned long long head;   // bytes taken from the end
    int32_t avail;             // chunks in the free ring
    uint32_t pushed, popped;   // ring positions
    uint32_t pad;
};

struct WfaArgs {
    const uint8_t *pat, *txt;
    const uint64_t *ppat, *ptxt;  // the same arenas at 2 bits per base (32 bases per word)
    const WfaPairDev *pairs;
    const int32_t *order;
    int32_t n;
    const int32_t *order_long;  // pairs each run on a whole CTA first, n_long of them
    int32_t n_long;
    uint8_t *pool;
    int64_t pool_bytes;
    WfaPoolCtl *ctl;
    int32_t *free_ring;   // chunks given back by finished pairs: chunk number + 1, 0 = empty slot
    // at least the chunks of the pool; 0: one pair alone, in as little of the pool as it can do with
    // (wavefronts trimmed from the start, memory taken in exact pieces that are not given back)
    uint32_t free_slots;
    int64_t *ctab;
    char *ops;
    WfaOutDev *out;
    int32_t *queue;       // [0] next position of `order`, [1] pairs running, [3] pairs started,
                          // [q_long] next position of `order_long`
    int32_t q_long;
    int32_t n_all;        // pairs of the round, over all launches that share it
    WfaPen pen;
    int singletrack;
    int piggyback;        // medium / low memory: ring of recent scores + packed-CIGAR blocks
    int max_score_scope;
    int wide_width;       // warp kernel: a pair whose wavefront grows wider stops with WFA_WIDE (0 = never)
    int wide_width_tail;  // the same once every pair has started and at most wide_tail_pairs
    int wide_tail_pairs;  // still run on warps (<= wide_width)
    int wide_width_cta;   // the same for a pair on a whole CTA: the width that always stops it,
    int wide_tail_cta;    // and the one of the tail
};

// Pool bytes are taken and given back in chunks of this size.
constexpr int64_t WFA_CHUNK = 256 << 10;
// Computing threads of the kernel's CTAs, beside a planning warp: WFA_CTA (four CTAs fit an SM,
// three in the piggyback modes, whose trips need the registers: 2,048 pairs 36.7 against 39.3 ms
// with four), or WFA_BIG_CTA (one per SM; sixteen warps with the planner's) for the pairs that
// would outlast their batch on the small ones.
constexpr int WFA_CTA = 128, WFA_BIG_CTA = 480;

cudaError_t launch_wfa(const WfaArgs &a, int threads, int ctas, cudaStream_t st);
// The cluster kernel (high memory: standard and Singletrack): one cluster of `cl` CTAs per
// pair, the diagonals of a wavefront spread over all of its threads; `clusters` clusters
// take the pairs of a.order in turn.
cudaError_t launch_wfa_wide(const WfaArgs &a, int clusters, int cl, cudaStream_t st);
// Clusters of `cl` CTAs of the cluster kernel that fit on the device at once for a score
// scope (0 if none, or if the scope is too large for the kernel's header ring).
int wfa_wide_clusters(int cl, const WfaPen &pen, int scope);
// 2-bit copies of the pattern and text arenas (A=0, C=1, G=2, T=3, any other byte 0), and
// the per-pair flag that the pair's sequences are uppercase ACGT only.
cudaError_t launch_wfa_pack(const uint8_t *pat, int64_t pbytes, uint64_t *ppat, const uint8_t *txt, int64_t tbytes,
                            uint64_t *ptxt, WfaPairDev *pairs, int n, cudaStream_t st);
int wfa_occupancy(bool piggyback, int threads, const WfaPen &pen, int scope);

}  // namespace aw
