// dp_kernels.cu - sm_100a kernels of the level-synchronous join-order DP and
// the host engine that sequences them.
//
// Per level k = 2..n (the reference's host loop gpuqo_dpsub_common.cu:295-342):
//   k_filter  - combinadic unrank + Gosper stepping over the C(n,k) candidate
//               sets, connectivity test against the adjacency in shared
//               memory, stream compaction of the connected sets in shared
//               memory (one global atomic per 32 survivors).  Replaces the
//               reference's unrankFilteredDPSubKernel + thrust::remove
//               (gpuqo_dpsub_filtered_kernels.cuh:31-109, gpuqo_dpsub_filtered.cu:120).
//   k_eval    - one warp per connected set: csg-cmp candidates (all subsets,
//               or MPDP biconnected-block candidates), CCC queue so that cost
//               evaluations run warp-full, join cost, warp min-reduction on
//               (cost, enumeration index) and a direct dense-memo write.
//               Replaces evaluateFilteredDPSubKernel + the scratchpad scatter
//               into the hash table (gpuqo_dpsub_filtered_kernels.cuh:152-333,
//               gpuqo_dpsub_common.cu:152-166).
//   k_ovf_*   - sets whose candidate count exceeds one warp's share are split
//               into chunks over all warps; each chunk folds its best into a
//               64-bit atomicMin on (ordered cost << 32 | index); a finalize
//               pass re-derives the winner and writes the memo.
// After the last level k_extract walks the memo back-pointers on the device
// and the host copies one small node array (replaces dpsub_buildQueryTree's
// per-node lookups, gpuqo_query_tree.cuh:47-71).
//
// Tie rule: the reference's CPU engines keep the FIRST strict minimum of
// cost.total in their enumeration order (gpuqo_cpu_common.cuh:202).  Keys are
// (ordered cost, enumeration index), so the lexicographic minimum is that
// element; a NaN cost never replaces, and a NaN first candidate is kept, as
// with the reference's '<' comparisons.
//
// The launch sequence of one query is captured once into a CUDA graph per
// (n, mode, ccc) and replayed; the host never synchronises between levels.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "dp_device.cuh"
#include "dp_engine.h"
#include "dp_barrier.cuh"
#include "dp_general.cuh"
#include "gpuqo_b200.h"

extern "C" int gpuqo_b200_persistent;
extern "C" int gpuqo_b200_barrier_poll_limit;
extern "C" int gpuqo_b200_device_memory_mb;

namespace gqb {

constexpr int kBlock = 256;
constexpr int kWarpsPerBlock = kBlock / 32;
constexpr uint32_t kFull = 0xFFFFFFFFu;
// candidates per warp above which a set goes to the chunked overflow path
constexpr uint32_t kOvfLimit = 32u * 64u;
// candidates per overflow chunk
constexpr uint32_t kChunk = 32u * 64u;
constexpr int kQueueWords = 64 * 3;    // per-warp CCC queue: 64 x (p, L, R)

// units of chunked work of a set with P candidates: plain DPsub costs a split
// and its mirror together (eval_range_dpsub), so its P candidates are P / 2
// units; MPDP candidates are one unit each
__host__ __device__ __forceinline__ uint32_t ovf_work(int mode, uint32_t P) { return mode == kModeDpsub ? P / 2u : P; }

struct LevelCounters {
    uint32_t n_sets;                   // connected sets found by k_filter
    uint32_t chunk_next;               // overflow work counter
    unsigned long long ovf_packed;     // (n_ovf << 40) | n_chunks
    uint32_t n_fb;                     // sets sent to the exact-order fallback
    uint32_t pad;
};

struct GlobalCounters {
    unsigned long long evaluated_pairs;
};

struct DevArena {
    float4 *memo = nullptr;            // [2^n] rows, startup, total, width bits
    uint32_t *memo_left = nullptr;     // [2^n] left (outer) set of the best join
    uint32_t *sets = nullptr;          // [maxC] connected sets of the current level
    uint32_t *sets2 = nullptr;         // [maxC] second level list (levels alternate)
    uint32_t *seen = nullptr;          // [2^n bits] extension dedup bitmap
    uint32_t *ovf_set = nullptr;       // [maxC]
    uint32_t *ovf_P = nullptr;         // [maxC]
    uint32_t *ovf_off = nullptr;       // [maxC] first chunk id
    unsigned long long *ovf_key = nullptr;   // [maxC]
    unsigned long long *ovf_first = nullptr; // [maxC]
    LevelCounters *lvl = nullptr;      // [33]
    GlobalCounters *glob = nullptr;
    uint32_t *blob = nullptr;          // device planner info
    uint32_t *binom = nullptr;         // [33*33] C(i, j)
    TreeNode *tree = nullptr;          // [64]
    int *tree_n = nullptr;
    unsigned *bar = nullptr;           // grid barrier of the persistent kernel: arrivals, generation, error
    // DPsize only (allocated on its first use)
    uint32_t *pos = nullptr;           // [2^n] place of a set in its level list
    uint32_t *bmask = nullptr;         // [maxC] per set of the previous level: places of its discoveries
    uint32_t *bstart = nullptr;        // [maxC] exclusive prefix of the mask popcounts
    uint32_t *tile_sum = nullptr;      // [maxC / kScanTile + 2]
    unsigned long long *disc = nullptr;   // [maxC] discovery key of each set of the level
    uint32_t *level1 = nullptr;        // [32] the level-1 list (place of each relation)
};

// ---------------------------------------------------------------------------
// k_filter: connected k-subsets of n relations
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t unrank_ksubset(uint64_t r, int n, int k, const uint32_t *binom) {
    // r-th k-subset of {0..n-1} in increasing integer order
    uint32_t s = 0;
    int kk = k;
    for (int pos = n - 1; pos >= 0 && kk > 0; pos--) {
        uint32_t c = binom[pos * 33 + kk];     // kk-subsets of {0..pos-1}
        if (r >= c) {
            s |= 1u << pos;
            r -= c;
            kk--;
        }
    }
    return s;
}

__device__ __forceinline__ uint32_t gosper_next(uint32_t v) {
    uint32_t t = v | (v - 1u);
    return (t + 1u) | (((~t & (0u - ~t)) - 1u) >> __ffs(v));
}

__global__ void __launch_bounds__(kBlock) k_filter(const uint32_t *__restrict__ blob, const uint32_t *__restrict__ binom_g,
                                                   int n, int k, unsigned long long total, uint32_t per_thread,
                                                   uint32_t *__restrict__ out_sets, LevelCounters *__restrict__ lc) {
    __shared__ uint32_t adj[kMaxRels];
    __shared__ uint32_t binom[33 * 33];
    __shared__ uint32_t stage[kWarpsPerBlock][64];
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob);
    for (int i = threadIdx.x; i < kMaxRels; i += blockDim.x) adj[i] = (i < n) ? h->adj[i] : 0u;
    for (int i = threadIdx.x; i < 33 * 33; i += blockDim.x) binom[i] = binom_g[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *st = stage[warp];
    uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t r0 = tid * per_thread;
    uint64_t r1 = r0 + per_thread < total ? r0 + per_thread : total;
    uint32_t s = r0 < total ? unrank_ksubset(r0, n, k, binom) : 0u;
    uint32_t cnt = 0;
    for (uint32_t j = 0; j < per_thread; j++) {
        uint64_t r = r0 + j;
        bool has = r < r1;
        bool ok = has && is_connected(s, adj);
        uint32_t m = __ballot_sync(kFull, ok);
        if (ok) st[cnt + __popc(m & ((1u << lane) - 1u))] = s;
        cnt += __popc(m);
        __syncwarp();
        if (cnt >= 32) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&lc->n_sets, 32u);
            base = __shfl_sync(kFull, base, 0);
            out_sets[base + lane] = st[lane];
            __syncwarp();
            if (lane < cnt - 32) st[lane] = st[32 + lane];
            cnt -= 32;
            __syncwarp();
        }
        if (has && r + 1 < r1) s = gosper_next(s);
    }
    if (cnt > 0) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&lc->n_sets, cnt);
        base = __shfl_sync(kFull, base, 0);
        if (lane < cnt) out_sets[base + lane] = st[lane];
    }
}

// ---------------------------------------------------------------------------
// k_level_sets: the connected k-sets, by whichever enumeration is cheaper for
// this level (decided on the device from the previous level's count):
//   * extension: every connected (k-1)-set plus each of its neighbours; a
//     test-and-set bitmap over all 2^n sets keeps the first producer of each
//     k-set (work ~ count(k-1) * |neighbours|, for sparse graphs far below
//     C(n,k));
//   * filter: combinadic unrank + Gosper stepping over all C(n,k) subsets with
//     the connectivity test (as k_filter; dense graphs).
// Both produce the same set of connected k-sets; their order in the level list
// does not affect the result (each set's best join is computed independently).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) k_level_sets(const uint32_t *__restrict__ blob,
                                                       const uint32_t *__restrict__ binom_g, int n, int k,
                                                       unsigned long long total, uint32_t per_thread,
                                                       const uint32_t *__restrict__ prev_sets,
                                                       const LevelCounters *__restrict__ prev_lc,
                                                       uint32_t *__restrict__ bitmap, uint32_t *__restrict__ out_sets,
                                                       LevelCounters *__restrict__ lc) {
    __shared__ uint32_t adj[kMaxRels];
    __shared__ uint32_t binom[33 * 33];
    __shared__ uint32_t stage[kWarpsPerBlock][64];
    const uint32_t c_prev = (k == 2) ? (uint32_t)n : __ldcg(&prev_lc->n_sets);
    // per candidate the extension costs a neighbourhood scan share plus one
    // L2 atomic; the filter a Gosper step plus a short connectivity test
    const bool use_ext = (uint64_t)c_prev * (uint64_t)(k + 4 * (n - k + 1)) < total * 3ull;
    // the grid is sized for the filter; the extension needs one thread per
    // set of the previous level, so surplus blocks leave at once
    if (use_ext && (uint64_t)blockIdx.x * blockDim.x >= (uint64_t)c_prev) return;
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob);
    for (int i = threadIdx.x; i < kMaxRels; i += blockDim.x) adj[i] = (i < n) ? h->adj[i] : 0u;
    if (!use_ext)
        for (int i = threadIdx.x; i < 33 * 33; i += blockDim.x) binom[i] = binom_g[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *st = stage[warp];
    uint32_t cnt = 0;
    auto emit = [&](bool ok, uint32_t s) {
        uint32_t m = __ballot_sync(kFull, ok);
        if (ok) st[cnt + __popc(m & ((1u << lane) - 1u))] = s;
        cnt += __popc(m);
        __syncwarp();
        if (cnt >= 32) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&lc->n_sets, 32u);
            base = __shfl_sync(kFull, base, 0);
            out_sets[base + lane] = st[lane];
            __syncwarp();
            if (lane < cnt - 32) st[lane] = st[32 + lane];
            cnt -= 32;
            __syncwarp();
        }
    };
    if (use_ext) {
        const uint32_t used_blocks = (uint32_t)min((uint64_t)gridDim.x, ((uint64_t)c_prev + blockDim.x - 1) / blockDim.x);
        const uint32_t nthreads = used_blocks * blockDim.x;
        const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
        // warp-uniform trip count over the previous level
        const uint32_t rounds = (c_prev + nthreads - 1u) / nthreads;
        for (uint32_t r = 0; r < rounds; r++) {
            const uint32_t idx = tid + r * nthreads;
            uint32_t S = 0u, N = 0u;
            if (idx < c_prev) {
                S = (k == 2) ? (1u << idx) : __ldcg(prev_sets + idx);
                uint32_t x = S;
                while (x) {
                    int v = __ffs(x) - 1;
                    x &= x - 1u;
                    N |= adj[v];
                }
                N &= ~S;
            }
            const int deg = __popc(N);
            const int maxdeg = (int)__reduce_max_sync(kFull, (uint32_t)deg);
            for (int j = 0; j < maxdeg; j++) {
                bool ok = false;
                uint32_t T = 0u;
                if (j < deg) {
                    const uint32_t bitv = N & (0u - N);
                    N ^= bitv;
                    T = S | bitv;
                    const uint32_t bm = 1u << (T & 31u);
                    ok = !(atomicOr(&bitmap[T >> 5], bm) & bm);
                }
                emit(ok, T);
            }
        }
    } else {
        uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
        uint64_t r0 = tid * per_thread;
        uint64_t r1 = r0 + per_thread < total ? r0 + per_thread : total;
        uint32_t s = r0 < total ? unrank_ksubset(r0, n, k, binom) : 0u;
        for (uint32_t j = 0; j < per_thread; j++) {
            uint64_t r = r0 + j;
            bool has = r < r1;
            bool ok = has && is_connected(s, adj);
            emit(ok, s);
            if (has && r + 1 < r1) s = gosper_next(s);
        }
    }
    if (cnt > 0) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&lc->n_sets, cnt);
        base = __shfl_sync(kFull, base, 0);
        if (lane < cnt) out_sets[base + lane] = st[lane];
    }
}

// ---------------------------------------------------------------------------
// candidate enumeration + evaluation shared by k_eval / k_ovf_chunks
// ---------------------------------------------------------------------------
// A lane's first strict minimum over the candidates it costed.  The NaN rule
// (a NaN first candidate is kept) needs the lowest index of all candidates and
// of those with a NaN cost; NaN costs are rare, so a candidate pays one
// minimum and one untaken branch for it.
struct LaneBest {
    unsigned long long key;
    RelVal val;
    uint32_t left;
    uint32_t first_p;             // lowest index of a valid candidate
    uint32_t nan_p;               // lowest index of one with a NaN cost
    RelVal nan_val;
    uint32_t nan_left;
    uint32_t n_valid;

    __device__ __forceinline__ void init() {
        key = ~0ull;
        left = 0;
        first_p = kFull;
        nan_p = kFull;
        nan_left = 0;
        n_valid = 0;
    }
    __device__ __forceinline__ bool first_nan() const { return nan_p != kFull && nan_p == first_p; }
};

// one valid candidate p = (outer L, inner side) with its cost: the lane keeps
// its first strict minimum (key (ordered cost, p))
__device__ __forceinline__ void best_update(LaneBest &best, uint32_t p, uint32_t L, const RelVal &out) {
    best.n_valid++;
    best.first_p = min(best.first_p, p);
    if (__builtin_expect(isnan(out.total), 0)) {
        if (p < best.nan_p) {
            best.nan_p = p;
            best.nan_val = out;
            best.nan_left = L;
        }
        return;
    }
    const unsigned long long key = ((unsigned long long)ord_float(out.total) << 32) | p;
    if (key < best.key) {
        best.key = key;
        best.val = out;
        best.left = L;
    }
}

__device__ __forceinline__ void evaluate_pair(const DevInfoView &d, const float4 *memo, uint32_t p, uint32_t L,
                                              uint32_t R, LaneBest &b) {
    const RelVal l = load_rel(memo, L, d.h->hz_packed);
    const RelVal r = load_rel(memo, R, d.h->hz_packed);
    best_update(b, p, L, join_eval(d, L, l, R, r));
}

// A valid split (L, R) of a plain-DPsub set and its mirror (R, L), costed in
// one pass (join_eval_mirror); p and pm are their indices in the reference's
// enumeration order.
__device__ __forceinline__ void evaluate_mirror(const DevInfoView &d, const float4 *memo, uint32_t p, uint32_t pm,
                                                uint32_t L, uint32_t R, LaneBest &b) {
    const RelVal l = load_rel(memo, L, d.h->hz_packed);
    const RelVal r = load_rel(memo, R, d.h->hz_packed);
    RelVal out_lr, out_rl;
    join_eval_mirror(d, L, l, R, r, out_lr, out_rl);
    best_update(b, p, L, out_lr);
    best_update(b, pm, R, out_rl);
}

// Plain DPsub over mirror pairs: the reference visits L = pdep(p + 1, S) for
// p = 0 .. P - 1 (P = 2^|S| - 2, gpuqo_cpu_dpsub.cu:32-78), and candidate
// P - 1 - p is the complement of candidate p.  Lanes take contiguous slices
// of [lo, hi) within [0, P / 2); each h names the split L = pdep(h + 1, S)
// and its mirror, both connected or neither, costed together and keyed by
// their own indices h and P - 1 - h.  With ccc the valid splits go through
// the per-warp queue and are costed 32 at a time (the reference's CCC,
// gpuqo_dpsub.cuh:193-259, as a compaction queue).
__device__ __forceinline__ void eval_range_dpsub(const DevInfoView &d, const uint32_t *adj, uint32_t S, uint32_t P,
                                                 uint32_t lo, uint32_t hi, const float4 *memo, uint32_t *q,
                                                 bool ccc, LaneBest &best) {
    const int lane = threadIdx.x & 31;
    const uint32_t span = hi - lo;
    const uint32_t per = (span + 31u) / 32u;
    uint32_t my_lo = lo + per * lane;
    if (my_lo > hi) my_lo = hi;
    const uint32_t my_hi = my_lo + per < hi ? my_lo + per : hi;
    uint32_t h = my_lo;
    uint32_t L = h < my_hi ? pdep32(h + 1u, S) : 0u;
    int qn = 0;   // warp-uniform queue length
    while (__any_sync(kFull, h < my_hi)) {
        const bool has = h < my_hi;
        bool valid = false;
        uint32_t cl = 0, cr = 0;
        if (has) {
            cl = L;
            cr = S ^ L;
            valid = is_connected(cl, adj) && is_connected(cr, adj);
            L = next_subset(L, S);
        }
        const uint32_t ch = h;
        if (has) h++;
        if (!ccc) {
            if (valid) evaluate_mirror(d, memo, ch, P - 1u - ch, cl, cr, best);
            continue;
        }
        const uint32_t m = __ballot_sync(kFull, valid);
        if (valid) {
            const int pos = qn + __popc(m & ((1u << lane) - 1u));
            q[pos * 3 + 0] = ch;
            q[pos * 3 + 1] = cl;
            q[pos * 3 + 2] = cr;
        }
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
            const int pos = qn - 32 + lane;
            const uint32_t eh = q[pos * 3 + 0], el = q[pos * 3 + 1], er = q[pos * 3 + 2];
            __syncwarp();
            qn -= 32;
            evaluate_mirror(d, memo, eh, P - 1u - eh, el, er, best);
        }
    }
    if (ccc && qn > 0) {
        __syncwarp();
        if (lane < qn) evaluate_mirror(d, memo, q[lane * 3 + 0], P - 1u - q[lane * 3 + 0], q[lane * 3 + 1],
                                       q[lane * 3 + 2], best);
    }
    __syncwarp();
}

// Enumerates candidate indices [lo, hi) of set S (lanes take contiguous
// slices), tests each candidate, and evaluates the valid ones.  With ccc the
// valid candidates go through a per-warp queue and are evaluated 32 at a time
// (the reference's CCC, gpuqo_dpsub.cuh:193-259, as a compaction queue).
template <int MODE>
__device__ __forceinline__ void eval_range(const DevInfoView &d, const uint32_t *adj, uint32_t S, const Blocks &B,
                                           uint32_t lo, uint32_t hi, const float4 *memo, uint32_t *q, bool ccc,
                                           LaneBest &best) {
    const int lane = threadIdx.x & 31;
    uint32_t span = hi - lo;
    uint32_t per = (span + 31u) / 32u;
    uint32_t my_lo = lo + per * lane;
    uint32_t my_hi = my_lo + per < hi ? my_lo + per : hi;
    if (my_lo > hi) my_lo = hi;
    uint32_t p = my_lo;
    // iterator state
    uint32_t L = 0;           // MODE 0: current left subset
    int b = 0;                // MODE 1: block index
    uint32_t lb = 0;          // MODE 1: current subset of block b
    uint32_t key = 0;         // MODE 1: the reference's index of the candidate
    CycleCache cc;            // MODE 1: arcs of the current cycle block
    if (p < my_hi) {
        if (MODE == kModeDpsub) {
            L = pdep32(p + 1u, S);
        } else {
            // p counts enumerated candidates (Blocks::eprefix); cycle blocks
            // decode their arcs per candidate, other blocks walk nextSubset
            while (b + 1 < B.nb && B.eprefix[b + 1] <= p) b++;
            if (!((B.cyc >> b) & 1u)) lb = pdep32(p - B.eprefix[b] + 1u, B.mask[b]);
        }
    }
    int qn = 0;   // warp-uniform queue length
    while (__any_sync(kFull, p < my_hi)) {
        bool has = p < my_hi;
        bool valid = false;
        uint32_t cl = 0, cr = 0;
        if (has) {
            if (MODE == kModeDpsub) {
                cl = L;
                cr = S ^ L;
                valid = is_connected(cl, adj) && is_connected(cr, adj);
                L = next_subset(L, S);
            } else {
                const uint32_t blk = B.mask[b];
                const bool cyc = (B.cyc >> b) & 1u;
                if (cyc) lb = cached_arc(cc, S, b, blk, adj, p - B.eprefix[b]);
                uint32_t rb = blk ^ lb;
                if (cyc && blk == S) {   // the set is the cycle: arc and complement
                    cl = lb;
                    cr = rb;
                } else {
                    cl = grow(lowest(lb), S & ~rb, adj);
                    cr = grow(lowest(rb), S & ~lb, adj);
                }
                valid = (cl | cr) == S;
                // the reference's index of this candidate (Blocks::prefix space)
                key = B.prefix[b] + (cyc ? pext32(lb, blk) - 1u : p - B.eprefix[b]);
                if (p + 1u < B.eprefix[b + 1]) {
                    if (!cyc) lb = next_subset(lb, blk);
                } else if (b + 1 < B.nb) {
                    b++;
                    lb = lowest(B.mask[b]);
                }
            }
        }
        uint32_t cp = (MODE == kModeMpdp) ? key : p;
        if (MODE == kModeMpdp && valid) cp = key_index(*d.h, key, cl, S);
        if (has) p++;
        if (!ccc) {
            if (valid) evaluate_pair(d, memo, cp, cl, cr, best);
            continue;
        }
        uint32_t m = __ballot_sync(kFull, valid);
        if (valid) {
            int pos = qn + __popc(m & ((1u << lane) - 1u));
            q[pos * 3 + 0] = cp;
            q[pos * 3 + 1] = cl;
            q[pos * 3 + 2] = cr;
        }
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
            int pos = qn - 32 + lane;
            uint32_t ep = q[pos * 3 + 0], el = q[pos * 3 + 1], er = q[pos * 3 + 2];
            __syncwarp();
            qn -= 32;
            evaluate_pair(d, memo, ep, el, er, best);
        }
    }
    if (ccc && qn > 0) {
        __syncwarp();
        if (lane < qn) evaluate_pair(d, memo, q[lane * 3 + 0], q[lane * 3 + 1], q[lane * 3 + 2], best);
    }
    __syncwarp();
}

struct WarpWinner {
    bool is_writer;
    bool use_nan;
};

__device__ __forceinline__ WarpWinner warp_winner(const LaneBest &b, unsigned long long &min_key,
                                                  unsigned long long &first_key) {
    uint32_t kh = (uint32_t)(b.key >> 32), kl = (uint32_t)b.key;
    uint32_t mh = __reduce_min_sync(kFull, kh);
    uint32_t ml = __reduce_min_sync(kFull, kh == mh ? kl : kFull);
    uint32_t mf = __reduce_min_sync(kFull, b.first_p);
    bool nan_first = (b.first_p == mf) && b.first_nan();
    unsigned nm = __ballot_sync(kFull, nan_first);
    min_key = ((unsigned long long)mh << 32) | ml;
    first_key = ((unsigned long long)mf << 1) | (nm ? 1ull : 0ull);
    WarpWinner w;
    if (nm) {
        w.is_writer = nan_first;
        w.use_nan = true;
    } else {
        w.is_writer = (b.key == min_key) && (b.key != ~0ull);
        w.use_nan = false;
    }
    return w;
}

__device__ __forceinline__ void memo_write(const DevHeader &h, float4 *memo, uint32_t *memo_left, uint32_t S,
                                           const RelVal &v, uint32_t left) {
    memo[S] = make_float4(v.rows, v.startup, v.total, __uint_as_float(memo_width_word(h, v.rows, v.width)));
    memo_left[S] = left;
}

__device__ __forceinline__ void load_blob_to_smem(const uint32_t *blob, uint32_t words, uint32_t *sm) {
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) sm[i] = blob[i];
    __syncthreads();
}

// ---------------------------------------------------------------------------
// k_eval: one warp per connected set
// ---------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(kBlock) k_eval(const uint32_t *__restrict__ blob, uint32_t blob_words, int k,
                                                 const uint32_t *__restrict__ sets, LevelCounters *__restrict__ lc,
                                                 float4 *__restrict__ memo, uint32_t *__restrict__ memo_left,
                                                 uint32_t *__restrict__ ovf_set, uint32_t *__restrict__ ovf_P,
                                                 uint32_t *__restrict__ ovf_off,
                                                 unsigned long long *__restrict__ ovf_key,
                                                 unsigned long long *__restrict__ ovf_first,
                                                 GlobalCounters *__restrict__ glob, int ccc,
                                                 const uint32_t *__restrict__ count_ptr = nullptr) {
    const uint32_t count = count_ptr ? *count_ptr : lc->n_sets;
    if (count == 0u) return;
    extern __shared__ __align__(16) uint32_t sm[];
    load_blob_to_smem(blob, blob_words, sm);
    const DevInfoView d = make_view(sm);
    const uint32_t *adj = d.h->adj;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *q = sm + ((blob_words + 3u) & ~3u) + warp * kQueueWords;
    const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
    unsigned long long pairs = 0;
    Blocks B;
    B.nb = 0;
    for (uint32_t i = blockIdx.x * kWarpsPerBlock + warp; i < count; i += nwarps) {
        const uint32_t S = sets[i];
        uint32_t P;
        if (MODE == kModeDpsub) {
            P = (1u << k) - 2u;
        } else {
            find_blocks(S, adj, B);
            P = B.etotal;
        }
        if (P > kOvfLimit) {
            if (lane == 0) {
                uint32_t nch = (ovf_work(MODE, P) + kChunk - 1u) / kChunk;
                unsigned long long old = atomicAdd(&lc->ovf_packed, (1ull << 40) | (unsigned long long)nch);
                uint32_t idx = (uint32_t)(old >> 40);
                ovf_set[idx] = S;
                ovf_P[idx] = P;
                ovf_off[idx] = (uint32_t)(old & 0xFFFFFFFFFFull);
                ovf_key[idx] = ~0ull;
                ovf_first[idx] = ~0ull;
            }
            continue;
        }
        LaneBest best;
        best.init();
        if constexpr (MODE == kModeDpsub) eval_range_dpsub(d, adj, S, P, 0u, P / 2u, memo, q, ccc != 0, best);
        else eval_range<MODE>(d, adj, S, B, 0u, P, memo, q, ccc != 0, best);
        unsigned long long mk, fk;
        WarpWinner w = warp_winner(best, mk, fk);
        if (w.is_writer) {
            if (w.use_nan) memo_write(*d.h, memo, memo_left, S, best.nan_val, best.nan_left);
            else memo_write(*d.h, memo, memo_left, S, best.val, best.left);
        }
        pairs += best.n_valid;
    }
    pairs = __reduce_add_sync(kFull, (uint32_t)pairs);
    if (lane == 0 && pairs) atomicAdd(&glob->evaluated_pairs, pairs);
}

// ---------------------------------------------------------------------------
// k_eval_mpdp: MPDP with G lanes per connected set (32/G sets per warp).
// G is picked on the device from the level's set count so that small levels
// still fill the GPU and large levels do not pay the per-set block search 32
// times per warp.  Lanes of a group take candidates p = g, g+G, ...; the loop
// runs the warp's maximum trip count so the group reductions can use
// full-warp shuffles.
// ---------------------------------------------------------------------------
template <int G>
__device__ __forceinline__ void mpdp_groups(const DevInfoView &d, const uint32_t *adj, uint32_t first_set,
                                            uint32_t stride_sets, const uint32_t *sets, uint32_t count,
                                            LevelCounters *lc, float4 *memo, uint32_t *memo_left,
                                            uint32_t *ovf_set, uint32_t *ovf_P, uint32_t *ovf_off,
                                            unsigned long long *ovf_key, unsigned long long *ovf_first,
                                            unsigned long long &pairs) {
    const int lane = threadIdx.x & 31;
    const int grp = lane / G, gl = lane % G;
    const uint32_t group_mask = (G == 32) ? kFull : (((1u << G) - 1u) << (grp * G));
    Blocks B;
    CycleCache cc;
    for (uint32_t base = first_set; base < count; base += stride_sets) {
        const uint32_t i = base + (uint32_t)grp;
        const bool has = i < count;
        const uint32_t S = has ? sets[i] : 0u;
        uint32_t P = 0;
        B.nb = 0;
        if (has) {
            find_blocks(S, adj, B);
            P = B.etotal;
        }
        __syncwarp();
        const bool ovf = has && P > kOvfLimit;
        if (ovf && gl == 0) {
            uint32_t nch = (P + kChunk - 1u) / kChunk;
            unsigned long long old = atomicAdd(&lc->ovf_packed, (1ull << 40) | (unsigned long long)nch);
            uint32_t idx = (uint32_t)(old >> 40);
            ovf_set[idx] = S;
            ovf_P[idx] = P;
            ovf_off[idx] = (uint32_t)(old & 0xFFFFFFFFFFull);
            ovf_key[idx] = ~0ull;
            ovf_first[idx] = ~0ull;
        }
        const uint32_t myP = (has && !ovf) ? P : 0u;
        const uint32_t iters = __reduce_max_sync(kFull, (myP + G - 1u) / G);
        LaneBest best;
        best.init();
        int b = 0;
        for (uint32_t it = 0; it < iters; it++) {
            const uint32_t p = (uint32_t)gl + it * G;
            if (p < myP) {
                uint32_t L, R;
                uint32_t key;
                if (mpdp_candidate(S, B, adj, p, b, L, R, key, cc))
                    evaluate_pair(d, memo, key_index(*d.h, key, L, S), L, R, best);
            }
        }
        // group reduction: min key, min first candidate (NaN rule)
        uint32_t kh = (uint32_t)(best.key >> 32), kl = (uint32_t)best.key, fp = best.first_p;
#pragma unroll
        for (int off = G / 2; off >= 1; off >>= 1) {
            uint32_t oh = __shfl_xor_sync(kFull, kh, off);
            uint32_t ol = __shfl_xor_sync(kFull, kl, off);
            uint32_t of = __shfl_xor_sync(kFull, fp, off);
            if (oh < kh || (oh == kh && ol < kl)) {
                kh = oh;
                kl = ol;
            }
            if (of < fp) fp = of;
        }
        const bool nan_first = has && !ovf && best.first_p == fp && best.first_nan();
        const unsigned nm = __ballot_sync(kFull, nan_first) & group_mask;
        const unsigned long long gkey = ((unsigned long long)kh << 32) | kl;
        if (has && !ovf) {
            if (nm) {
                if (nan_first) memo_write(*d.h, memo, memo_left, S, best.nan_val, best.nan_left);
            } else if (best.key == gkey && best.key != ~0ull) {
                memo_write(*d.h, memo, memo_left, S, best.val, best.left);
            }
        }
        pairs += best.n_valid;
    }
}

__global__ void __launch_bounds__(kBlock, 2) k_eval_mpdp(const uint32_t *__restrict__ blob, uint32_t blob_words,
                                                      const uint32_t *__restrict__ sets,
                                                      LevelCounters *__restrict__ lc, float4 *__restrict__ memo,
                                                      uint32_t *__restrict__ memo_left, uint32_t *__restrict__ ovf_set,
                                                      uint32_t *__restrict__ ovf_P, uint32_t *__restrict__ ovf_off,
                                                      unsigned long long *__restrict__ ovf_key,
                                                      unsigned long long *__restrict__ ovf_first,
                                                      GlobalCounters *__restrict__ glob, uint32_t target_lanes,
                                                      int max_group) {
    extern __shared__ __align__(16) uint32_t sm[];
    load_blob_to_smem(blob, blob_words, sm);
    const DevInfoView d = make_view(sm);
    const uint32_t *adj = d.h->adj;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t count = lc->n_sets;
    // lanes per set: enough lanes in flight to fill the GPU, no more than the
    // largest useful group for this level
    int G = 1;
    while (G < max_group && (uint64_t)count * (uint64_t)G < (uint64_t)target_lanes) G <<= 1;
    const uint32_t gwarp = blockIdx.x * kWarpsPerBlock + warp;
    const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
    unsigned long long pairs = 0;
    switch (G) {
#define GQB_G(g)                                                                                                  \
    case g:                                                                                                       \
        mpdp_groups<g>(d, adj, gwarp * (32 / g), nwarps * (32 / g), sets, count, lc, memo, memo_left, ovf_set,   \
                       ovf_P, ovf_off, ovf_key, ovf_first, pairs);                                                \
        break;
        GQB_G(1)
        GQB_G(2)
        GQB_G(4)
        GQB_G(8)
        GQB_G(16)
        GQB_G(32)
#undef GQB_G
    default:
        break;
    }
    pairs = __reduce_add_sync(kFull, (uint32_t)pairs);
    if (lane == 0 && pairs) atomicAdd(&glob->evaluated_pairs, pairs);
}

// ---------------------------------------------------------------------------
// MPDP on a tree-shaped query graph (star, snowflake, chain, and the
// contracted trees of IDP sub-problems), any relation numbering.
// A connected set S is a subtree; the reference's block search walks it from
// its lowest relation r, and every block is a bridge.  With the query tree
// rooted at r, every relation v of S but r is the child end of one split edge
// (v, parent of v), and removing it leaves S & sub_r[v] and the rest: no DFS,
// no search for the edge, one 8-byte table load per split.  Blocks are
// emitted in post-order of their child end, so the reference's enumeration
// index of a split is 2 * post_r(v) + (the lower end's side outer ? 0 : 1) with
//     post_r(v) = |S & before_r[v]| - |S & anc_r[v]| + |S & sub_r[v]| - 1
// (preorder rank minus depth plus subtree size minus one).
// ---------------------------------------------------------------------------
// what the classes of a query allow (one instantiation each, so that a kernel
// carries only the evaluation its queries take): kTreePlain
// DevHeader::tree_plain, kTreeMasked DevHeader::ec_masked, kTreeGeneral any
constexpr int kTreeGeneral = 0, kTreeMasked = 1, kTreePlain = 2;

__host__ __device__ __forceinline__ int tree_layout(const DevHeader &h) {
    return h.tree_plain ? kTreePlain : (h.ec_masked ? kTreeMasked : kTreeGeneral);
}

// one set's view of the tree tables: the rows of its lowest relation
struct TreeRows {
    const uint32_t *tab;   // tree tables
    const uint32_t *row;   // rows of the root
    int n;
};

__device__ __forceinline__ TreeRows tree_rows(const DevHeader &h, uint32_t S) {
    TreeRows t;
    t.tab = reinterpret_cast<const uint32_t *>(&h) + h.tree_tab;
    t.n = h.n;
    t.row = t.tab + (S ? t.tab[lowest_idx(S)] : 0u);
    return t;
}

// The reference's order of a split's two orientations: outer side L0 (the
// lower end's) and S - L0.  Block order: 2 * post_r(v) and the next; plain
// DPsub's: the subsets of S in increasing order, so the outer side itself.
__device__ __forceinline__ void tree_order(const TreeRows &t, uint32_t S, uint32_t v, uint32_t sub, uint32_t L0,
                                           uint32_t dpsub, uint32_t &p0, uint32_t &p1) {
    if (dpsub) {
        p0 = L0;
        p1 = S ^ L0;
    } else {
        const uint2 w = *reinterpret_cast<const uint2 *>(t.row + 2u * (uint32_t)t.n + 2u * v);
        p0 = 2u * (uint32_t)(__popc(S & w.x) - __popc(S & w.y) + __popc(S & sub) - 1);
        p1 = p0 + 1u;
    }
}

// A lane's best split of a set: (ordered cost, place in the reference's order)
// and the values the memo needs.  Equal costs are common (key joins leave the
// row counts of the larger side alone, so the order of several joins does not
// matter), hence the place is at hand and not computed on demand.
struct TreeBest {
    float total;
    uint32_t p;            // place, kFull: none yet
    uint32_t left;
    float rows, startup;
    uint32_t nan_p;        // lowest place of a candidate with a NaN cost, kFull: none

    __device__ __forceinline__ void init() {
        total = INFINITY;
        p = kFull;
        left = 0u;
        rows = startup = 0.0f;
        nan_p = kFull;
    }
};

// a NaN compares false and leaves the best as it is
__device__ __forceinline__ void tree_update(TreeBest &best, uint32_t p, uint32_t L, float rows, float startup,
                                            float total) {
    if (total < best.total || (total == best.total && p < best.p)) {
        best.total = total;
        best.p = p;
        best.left = L;
        best.rows = rows;
        best.startup = startup;
    }
}

__device__ __forceinline__ void tree_update_mirror(TreeBest &best, uint32_t S, uint32_t L0, uint32_t p0, uint32_t p1,
                                                   float rows0, float startup0, float total0, float rows1,
                                                   float startup1, float total1) {
    tree_update(best, p0, L0, rows0, startup0, total0);
    tree_update(best, p1, S ^ L0, rows1, startup1, total1);
    if (__builtin_expect(isnan(total0) || isnan(total1), 0)) {
        if (isnan(total0)) best.nan_p = min(best.nan_p, p0);
        if (isnan(total1)) best.nan_p = min(best.nan_p, p1);
    }
}

// both orientations of the split of S with the lower end's side L0 from the
// memo entries of that side (lv) and of the other (rv)
template <int LAYOUT>
__device__ __forceinline__ void tree_cost(const DevInfoView &d, const PlainParams &pp, const TreeRows &t, uint32_t S,
                                          uint32_t L0, uint32_t p0, uint32_t p1, uint32_t edge, const float4 lv,
                                          const float4 rv, TreeBest &best, int &width) {
    const DevHeader &h = *d.h;
    if (LAYOUT == kTreePlain) {
        const TreeEdge &e = reinterpret_cast<const TreeEdge *>(t.tab + tree_edge_off(t.n))[edge];
        JoinCost lr, rl;
        plain_mirror(pp, e.quals, e.sel_lo, e.sel_hi, lv, rv, lr, rl);
        width = (int)((__float_as_uint(lv.w) & kWidthMask) + (__float_as_uint(rv.w) & kWidthMask));
        tree_update_mirror(best, S, L0, p0, p1, lr.rows, lr.startup, lr.total, rl.rows, rl.startup, rl.total);
    } else {
        const RelVal l = unpack_rel(lv, h.hz_packed), r = unpack_rel(rv, h.hz_packed);
        RelVal o0, o1;
        const uint32_t classes =
            LAYOUT == kTreeMasked ? reinterpret_cast<const TreeEdge *>(t.tab + tree_edge_off(t.n))[edge].classes : 0u;
        join_eval_mirror_tree<LAYOUT == kTreeMasked>(d, L0, l, S ^ L0, r, classes, o0, o1);
        width = o0.width;
        tree_update_mirror(best, S, L0, p0, p1, o0.rows, o0.startup, o0.total, o1.rows, o1.startup, o1.total);
    }
}

// Some candidates of the warp's sets have a NaN cost (overflowed row
// estimates); the reference keeps such a one where it is a set's first.  The
// places of block order are 0 .. 2 (k - 1) - 1, so there it is the one at place
// 0; plain DPsub's first is the least outer side of all splits.  The lane that
// found it costs it again.  Returns whether the lane's group is settled.
template <int LAYOUT>
__device__ __noinline__ bool tree_nan_rule(const DevInfoView d, uint32_t S, bool has, int G, uint32_t nan_p,
                                           const float4 *memo, RelVal &out, uint32_t &left, bool &writer) {
    const DevHeader &h = *d.h;
    const TreeRows t = tree_rows(h, S);
    const int lane = (int)(threadIdx.x & 31u), gl = lane & (G - 1);
    uint32_t first = 0u;
    // the lane's own child ends, as tree_set deals them out
    uint32_t ends = has ? S & (S - 1u) : 0u;
    if (G == 32) {
        ends &= 1u << lane;
    } else {
        for (int i = 0; i < gl; i++) ends &= ends - 1u;
    }
    auto for_each_end = [&](auto body) {
        for (uint32_t x = ends; x;) {
            const uint32_t v = (uint32_t)lowest_idx(x);
            const uint2 e = *reinterpret_cast<const uint2 *>(t.row + 2u * v);
            body(v, e, (e.y & kTreeLower) ? S & e.x : S ^ (S & e.x));
            for (int i = 0; i < G; i++) x &= x - 1u;
        }
    };
    if (__any_sync(kFull, has && h.index_order != 0u)) {
        if (h.index_order != 0u) {
            first = kFull;
            for_each_end([&](uint32_t, uint2, uint32_t L0) { first = min(first, min(L0, S ^ L0)); });
        }
        for (int off = G >> 1; off >= 1; off >>= 1) first = min(first, __shfl_xor_sync(kFull, first, off));
    }
    writer = has && nan_p == first;   // kFull, no NaN, is no place
    const uint32_t writers = __ballot_sync(kFull, writer);
    if (writer) {
        uint32_t edge = 0u;
        for_each_end([&](uint32_t v, uint2 e, uint32_t L0) {
            uint32_t p0, p1;
            tree_order(t, S, v, e.x, L0, h.index_order, p0, p1);
            if (p0 != nan_p && p1 != nan_p) return;
            left = p0 == nan_p ? L0 : S ^ L0;
            edge = e.y & 31u;
        });
        const RelVal l = load_rel(memo, left, h.hz_packed), r = load_rel(memo, S ^ left, h.hz_packed);
        const uint32_t classes =
            LAYOUT == kTreeGeneral ? 0u : reinterpret_cast<const TreeEdge *>(t.tab + tree_edge_off(t.n))[edge].classes;
        out = join_eval_t<LAYOUT != kTreeGeneral>(d, left, l, S ^ left, r, classes);
    }
    return ((writers >> (lane - gl)) & (G == 32 ? kFull : (1u << G) - 1u)) != 0u;
}

// One set of k relations (has: the lane's group holds one) by a group of G
// lanes, G a power of two.  Lanes take the child ends by rank in S (a whole
// warp: by number); both memo entries of the next split are requested before
// the current one is costed.  The whole warp calls it, with the same k and G.
template <int LAYOUT>
__device__ __forceinline__ void tree_set(const DevInfoView &d, const PlainParams &pp, const TreeRows &t, uint32_t S,
                                         bool has, int k, int G, float4 *memo, uint32_t *memo_left) {
    const DevHeader &h = *d.h;
    const int lane = threadIdx.x & 31, gl = lane & (G - 1);
    uint32_t x = has ? S & (S - 1u) : 0u;
    if (G == 32) {
        x &= 1u << lane;   // at most 31 child ends: the lane's own relation
    } else {
        for (int i = 0; i < gl; i++) x &= x - 1u;
    }
    const int steps = G == 32 ? 1 : (k - 1 + G - 1) / G;
    TreeBest best;
    best.init();
    int width = 0;
    uint32_t p0 = 0u, p1 = 0u, L0 = 0u, edge = 0u;
    float4 lv = make_float4(0.f, 0.f, 0.f, 0.f), rv = lv;
    auto fetch = [&]() -> bool {
        if (x == 0u) return false;
        const uint32_t v = (uint32_t)lowest_idx(x);
        const uint2 e = *reinterpret_cast<const uint2 *>(t.row + 2u * v);
        const uint32_t comp = S & e.x;
        L0 = (e.y & kTreeLower) ? comp : S ^ comp;
        lv = __ldcg(memo + L0);
        rv = __ldcg(memo + (S ^ L0));
        edge = e.y & 31u;
        tree_order(t, S, v, e.x, L0, h.index_order, p0, p1);
        return true;
    };
    bool active = fetch();
    for (int j = 0; j < steps; j++) {
        const uint32_t c0 = p0, c1 = p1, cL = L0, ce = edge;
        const float4 clv = lv, crv = rv;
        const bool cact = active;
        active = false;
        if (j + 1 < steps) {
            for (int i = 0; i < G; i++) x &= x - 1u;
            active = fetch();
        }
        if (cact) tree_cost<LAYOUT>(d, pp, t, S, cL, c0, c1, ce, clv, crv, best, width);
    }
    uint32_t mh = best.p == kFull ? kFull : ord_float(best.total), ml = best.p;
    const uint32_t own = mh;
    if (G == 32) {
        const uint32_t w = __reduce_min_sync(kFull, mh);
        ml = __reduce_min_sync(kFull, mh == w ? ml : kFull);
        mh = w;
    } else {
        for (int off = G >> 1; off >= 1; off >>= 1) {
            const uint32_t oh = __shfl_xor_sync(kFull, mh, off), ol = __shfl_xor_sync(kFull, ml, off);
            if (oh < mh || (oh == mh && ol < ml)) {
                mh = oh;
                ml = ol;
            }
        }
    }
    bool win = has && best.p != kFull && own == mh && best.p == ml;
    if (__any_sync(kFull, best.nan_p != kFull)) {
        RelVal out;
        uint32_t left = 0u;
        bool writer = false;
        if (tree_nan_rule<LAYOUT>(d, S, has, G, best.nan_p, memo, out, left, writer)) win = false;
        if (writer) memo_write(h, memo, memo_left, S, out, left);
    }
    if (win) {
        const uint32_t word = LAYOUT == kTreePlain ? plain_width_word(h, best.rows, width)
                                                   : memo_width_word(h, best.rows, width);
        memo[S] = make_float4(best.rows, best.startup, best.total, __uint_as_float(word));
        memo_left[S] = best.left;
    }
}

// Lanes per set of a level of `count` sets of k relations with `lanes` lanes
// resident.  A warp-step (one split, both orientations) issues about kIssue
// instructions and takes kStep cycles; a set adds about one step of its own
// (list entry, reduction, memo entry).  The level takes the larger of its
// issue time and its longest lane's time; the smallest of the powers of two
// wins, the narrower group on ties.
__host__ __device__ __forceinline__ int tree_group(uint32_t count, int k, uint32_t lanes, uint32_t sms) {
    const float kIssue = 240.0f, kStep = 1500.0f;
    int best = 1;
    float best_t = 3.0e38f;
    for (int G = 1; G <= 32; G <<= 1) {
        const float steps = G == 32 ? 1.0f : (float)((k - 1 + G - 1) / G);
        const float warps = ceilf((float)count * (float)G / 32.0f);
        const float rounds = ceilf(warps * 32.0f / (float)lanes);
        const float issue = warps * (steps + 1.0f) * kIssue / (4.0f * (float)sms);
        const float chain = rounds * (steps + 1.0f) * kStep;
        const float t = issue > chain ? issue : chain;
        if (t < best_t) {
            best_t = t;
            best = G;
        }
        if (G >= k - 1) break;
    }
    return best;
}

template <int LAYOUT>
__device__ __forceinline__ void tree_level(const DevInfoView &d, const PlainParams &pp, uint32_t gwarp, uint32_t nwarps,
                                           const uint32_t *sets, uint32_t count, int k, int G, float4 *memo,
                                           uint32_t *memo_left) {
    const uint32_t per_warp = 32u / (uint32_t)G, grp = (threadIdx.x & 31u) / (uint32_t)G;
    for (uint32_t base = gwarp * per_warp; base < count; base += nwarps * per_warp) {
        const bool has = base + grp < count;
        const uint32_t S = has ? __ldcg(sets + base + grp) : 0u;
        tree_set<LAYOUT>(d, pp, tree_rows(*d.h, S), S, has, k, G, memo, memo_left);
    }
}

// one level per launch (gpuqo_b200_persistent = 0, no cooperative launch, or
// after a barrier timeout)
__global__ void __launch_bounds__(kBlock, 3) k_eval_tree(const uint32_t *__restrict__ blob, uint32_t blob_words, int k,
                                                      const uint32_t *__restrict__ sets,
                                                      LevelCounters *__restrict__ lc, float4 *__restrict__ memo,
                                                      uint32_t *__restrict__ memo_left,
                                                      GlobalCounters *__restrict__ glob) {
    extern __shared__ __align__(16) uint32_t sm[];
    load_blob_to_smem(blob, blob_words, sm);
    const DevInfoView d = make_view(sm);
    const uint32_t count = lc->n_sets;
    const uint32_t gwarp = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
    const int G = tree_group(count, k, nwarps * 32u, gridDim.x);
    const PlainParams pp = plain_params(*d.h);
    switch (tree_layout(*d.h)) {
    case kTreePlain:
        tree_level<kTreePlain>(d, pp, gwarp, nwarps, sets, count, k, G, memo, memo_left);
        break;
    case kTreeMasked:
        tree_level<kTreeMasked>(d, pp, gwarp, nwarps, sets, count, k, G, memo, memo_left);
        break;
    default:
        tree_level<kTreeGeneral>(d, pp, gwarp, nwarps, sets, count, k, G, memo, memo_left);
        break;
    }
    // every split edge, both orientations
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(&glob->evaluated_pairs, (unsigned long long)count * 2ull * (unsigned long long)(k - 1));
}

// ---------------------------------------------------------------------------
// k_dp_tree: the whole MPDP of a tree-shaped query in ONE persistent launch:
// cooperative, or for queries of narrow levels an ordinary launch of one
// thread-block cluster (or one block).  The planner info is staged in shared
// memory once; levels are separated by a barrier, and each phase evaluates
// level k while enumerating level k+1 (independent: the enumeration reads only
// level k's sets).  Data written by other blocks is read with ld.global.cg
// (L2), never through a possibly stale L1 line.
// The grid barrier spins a bounded number of times; on timeout it raises an
// error flag, every block leaves, and the host reruns the DP with per-level
// launches.  A cluster has the hardware's barrier.
// ---------------------------------------------------------------------------
// One enumeration phase (level k from the connected (k-1)-sets) of a
// tree-shaped query graph, each k-set once and without a dedup structure:
// adding a neighbour v to a connected set S of a tree makes v a leaf of
// T = S + v, and T is emitted only from the S whose added v is T's largest
// leaf.  T's other leaves are the leaves of S but the relation that v hangs
// off: with m1 > m2 the two largest leaves of S, a neighbour of m1 must exceed
// m2 and any other neighbour must exceed m1 (a single relation: itself).  So
// the extensions of S are one mask, counted and placed with one atomic per
// warp; the loop over the relations of S costs about 10 instructions each.
// near: the same with T's smallest leaf (m1 < m2 the two smallest, v below
// them), for memos beyond the caches (near_order).  The sets that one S emits,
// and those of the S next to it in the list, then share their high relations,
// so that the memo entries a warp reads and writes lie close together; by the
// largest leaf they share the low ones, and with them mostly the row of the
// tables that the warp reads (the row of a set's lowest relation).

// the relations v of the neighbours N of S whose addition emits S + v
template <class Adj>
__device__ __forceinline__ uint32_t tree_extension_mask(uint32_t S, uint32_t N, uint32_t leaves, bool near, Adj adj) {
    auto end = [&](uint32_t x) { return near ? lowest(x) : 1u << (31 - __clz(x)); };
    auto beyond = [&](uint32_t bit) { return near ? bit - 1u : ~((bit << 1) - 1u); };
    const uint32_t m1 = end(leaves), rest = leaves ^ m1;
    if (rest == 0u) return N & beyond(m1);                     // a single relation
    const uint32_t a1 = adj(lowest_idx(m1));
    return N & ((beyond(m1) & ~a1) | (beyond(end(rest)) & a1));
}

// the same from S alone (adj(v): neighbours of v)
template <class Adj>
__device__ __forceinline__ uint32_t tree_extensions(uint32_t S, bool near, Adj adj) {
    uint32_t N = 0u, leaves = 0u;
    for (uint32_t x = S; x; x &= x - 1u) {
        const uint32_t a = adj(lowest_idx(x)), in = a & S;
        N |= a;
        if ((in & (in - 1u)) == 0u) leaves |= x & (0u - x);   // S is connected: at least one neighbour in S
    }
    return S ? tree_extension_mask(S, N & ~S, leaves, near, adj) : 0u;
}

__device__ __forceinline__ void tree_enum_phase(const uint32_t *adj, int k, bool near, const uint32_t *prev_sets,
                                                uint32_t c_prev, uint32_t *out_sets, LevelCounters *lc) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nthreads = gridDim.x * blockDim.x;
    // from the far end of the grid: the first warps evaluate the first sets
    // of the level in the same phase, so small levels split the two jobs
    const uint32_t tid = nthreads - 1u - (blockIdx.x * blockDim.x + threadIdx.x);
    if (c_prev * 32u <= nthreads) {
        // a level that leaves warps idle: one warp per set and one lane per
        // relation, about 40 instructions instead of 10 per relation of the set
        const uint32_t i = tid >> 5;
        if (i >= c_prev) return;
        const uint32_t S = (k == 2) ? (1u << i) : __ldcg(prev_sets + i);
        const uint32_t a = ((S >> lane) & 1u) ? adj[lane] : 0u, in = a & S;
        const uint32_t leaves = __ballot_sync(kFull, a != 0u && (in & (in - 1u)) == 0u);
        const uint32_t ext =
            tree_extension_mask(S, __reduce_or_sync(kFull, a) & ~S, leaves, near, [&](int v) { return adj[v]; });
        uint32_t base = 0u;
        if (lane == 0u && ext) base = atomicAdd(&lc->n_sets, (uint32_t)__popc(ext));
        base = __shfl_sync(kFull, base, 0);
        if ((ext >> lane) & 1u) out_sets[base + (uint32_t)__popc(ext & ((1u << lane) - 1u))] = S | (1u << lane);
        return;
    }
    for (uint32_t first = tid & ~31u; first < c_prev; first += nthreads) {
        const uint32_t idx = first + (tid & 31u);
        const uint32_t S = idx < c_prev ? ((k == 2) ? (1u << idx) : __ldcg(prev_sets + idx)) : 0u;
        uint32_t ext = tree_extensions(S, near, [&](int v) { return adj[v]; });
        const uint32_t cnt = (uint32_t)__popc(ext);
        uint32_t incl = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(kFull, incl, off);
            if (lane >= (uint32_t)off) incl += o;
        }
        uint32_t base = 0u;
        if (lane == 31u && incl) base = atomicAdd(&lc->n_sets, incl);
        uint32_t at = __shfl_sync(kFull, base, 31) + incl - cnt;
        for (; ext; ext &= ext - 1u) out_sets[at++] = S | (ext & (0u - ext));
    }
}

// The plan, walked from the full set by one warp, level by level of the join
// tree: a lane per node reads its memo entry and outer side (about 0.35 us
// from L2), so the walk costs the plan's depth instead of its 2n - 1 nodes.
// Node 0 is the root; sets: 64 words of shared memory.
__device__ __forceinline__ void extract_plan(const float4 *memo, const uint32_t *memo_left, uint32_t full,
                                             uint32_t wmask, uint32_t *sets, TreeNode *out, int *n_out) {
    const uint32_t lane = threadIdx.x & 31u;
    if (lane == 0u) sets[0] = full;
    __syncwarp();
    uint32_t head = 0u, tail = 1u;
    while (head < tail) {
        const uint32_t me = head + lane;
        const bool has = me < tail;
        const uint32_t s = has ? sets[me] : 0u;
        TreeNode t;
        t.set = s;
        t.left = t.right = -1;
        uint32_t l = 0u;
        if (has) {
            const float4 v = __ldcg(memo + s);
            l = __ldcg(memo_left + s) & s;
            t.rows = v.x;
            t.startup = v.y;
            t.total = v.z;
            t.width = (int)(__float_as_uint(v.w) & wmask);
        }
        const bool join = has && popc(s) > 1 && l != 0u && l != s;
        const uint32_t joins = __ballot_sync(kFull, join);
        const uint32_t child = tail + 2u * (uint32_t)popc(joins & ((1u << lane) - 1u));
        if (join && child + 1u < 64u) {
            t.left = (int)child;
            t.right = (int)child + 1;
            sets[child] = l;
            sets[child + 1u] = s ^ l;
        }
        if (has) out[me] = t;
        head = min(tail, head + 32u);
        tail = min(tail + 2u * (uint32_t)popc(joins), 64u);
        __syncwarp();
    }
    if (lane == 0u) *n_out = (int)tail;
}

// Connected sets and lanes per set of every level, known on the host before
// the launch (a tree's connected subtrees are counted by size without listing
// them, tree_level_counts)
struct TreePlan {
    uint32_t count[33];
    uint8_t group[33];
    uint8_t near;                      // order of the lists (near_order)
};

// Bound: a warp-step (one split, both orientations) issues about 240
// instructions on a plain tree; wide levels are issue-bound, narrow ones wait
// for the chain list entry (about 700 cycles from L2) -> two memo entries (700)
// -> cost (500) -> reduction (300) -> memo entry (450) -> barrier (100 cycles in
// one block, 900 in a cluster of 8, 2000 over 296 blocks).  With the child end
// of a split read from the root's row, the sums over an edge's classes made on
// the host (TreeEdge), the extensions of a set as one mask, the order of a
// split at hand for equal costs, and grids no larger than the widest level
// needs, one cluster where that does: device time of star-22 (44.0 M pairs)
// 751 -> 387 us, snowflake-25 (3.2 M and 4.8 M pairs) 265 / 290 -> 139 us, key
// chain-30 203 -> 90 us, star-12 77 -> 47 us, star-6 38 -> 20 us.
// tree and tree_n are the host's (pinned): tree_n stays 0 when a barrier gives
// up.  blob may be the host's too: a few blocks read it faster than a copy
// ahead of the launch takes.
// MINB: blocks per SM the register budget is set for (2, 3 or 4: 128, 80 or 64
// registers; spill: 16 bytes with 3 blocks and general classes, 20 with 4
// blocks), chosen per query from its
// connected sets per level, the total over the relation count
// (Tuning::single_narrow_level_sets, Tuning::single_wide_level_sets); LAYOUT:
// the evaluation (tree_layout)
template <int MINB, int LAYOUT>
__global__ void __launch_bounds__(kBlock, MINB) k_dp_tree(const uint32_t *__restrict__ blob, uint32_t blob_words,
                                                       float4 *__restrict__ memo,
                                                       uint32_t *__restrict__ memo_left, uint32_t *__restrict__ setsA,
                                                       uint32_t *__restrict__ setsB, LevelCounters *__restrict__ lvl,
                                                       TreeNode *__restrict__ tree, int *__restrict__ tree_n,
                                                       unsigned *__restrict__ bar, unsigned bar_base,
                                                       const __grid_constant__ TreePlan plan, unsigned poll_limit) {
    extern __shared__ __align__(16) uint32_t sm[];
    const unsigned max_polls = barrier_polls(poll_limit);
    for (uint32_t i = threadIdx.x; i < blob_words / 4u; i += blockDim.x)
        reinterpret_cast<uint4 *>(sm)[i] = reinterpret_cast<const uint4 *>(blob)[i];
    __syncthreads();
    const DevInfoView d = make_view(sm);
    const int n = d.h->n;
    const uint32_t *adj = d.h->adj;
    const uint32_t gwarp = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
    const PlainParams pp = plain_params(*d.h);
    unsigned epoch = 0;   // grid barriers passed (thread 0)
    // one block, or a grid that is one cluster, synchronises in hardware; the
    // other variants never run as one
    const bool cluster = MINB == 2 && cluster_blocks() == gridDim.x;
    auto barrier = [&]() -> bool {
        if (MINB == 2 && cluster) {
            if (gridDim.x == 1u) __syncthreads();
            else cluster_barrier();
            return true;
        }
        return grid_barrier<true>(bar, epoch, max_polls, bar_base);
    };

    // phase 0: base relations (gpuqo_cpu_sequential.cu:80-92) and level-2 sets
    if (blockIdx.x == 0 && threadIdx.x < n) {
        const int i = threadIdx.x;
        memo[1u << i] = base_entry(*d.h, i);
        memo_left[1u << i] = 0u;
    }
    if (n >= 2) tree_enum_phase(adj, 2, plan.near != 0u, nullptr, (uint32_t)n, setsA, lvl + 2);
    if (!barrier()) return;
    for (int k = 2; k <= n; k++) {
        uint32_t *cur = (k & 1) ? setsB : setsA;
        uint32_t *nxt = (k & 1) ? setsA : setsB;
        const uint32_t count = plan.count[k];
        if (k < n) tree_enum_phase(adj, k + 1, plan.near != 0u, cur, count, nxt, lvl + k + 1);
        tree_level<LAYOUT>(d, pp, gwarp, nwarps, cur, count, k, plan.group[k], memo, memo_left);
        if (!barrier()) return;
    }
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        __shared__ uint32_t plan_sets[64];
        const uint32_t full = (n == 32) ? 0xFFFFFFFFu : ((1u << n) - 1u);
        extract_plan(memo, memo_left, full, d.h->hz_packed ? kWidthMask : 0xFFFFFFFFu, plan_sets, tree, tree_n);
        // the counters as the next launch expects them (nobody adds any more)
        for (int k = 2 + (int)threadIdx.x; k <= n; k += 32) lvl[k].n_sets = 0u;
    }
}

// ---------------------------------------------------------------------------
// k_ovf_chunks / k_ovf_finalize: large sets split over all warps
// ---------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(kBlock, 3) k_ovf_chunks(const uint32_t *__restrict__ blob, uint32_t blob_words, int k,
                                                       LevelCounters *__restrict__ lc, const float4 *__restrict__ memo,
                                                       const uint32_t *__restrict__ ovf_set,
                                                       const uint32_t *__restrict__ ovf_P,
                                                       const uint32_t *__restrict__ ovf_off,
                                                       unsigned long long *__restrict__ ovf_key,
                                                       unsigned long long *__restrict__ ovf_first,
                                                       GlobalCounters *__restrict__ glob, int ccc) {
    const unsigned long long packed = lc->ovf_packed;
    const uint32_t n_ovf = (uint32_t)(packed >> 40);
    const uint32_t n_chunks = (uint32_t)(packed & 0xFFFFFFFFFFull);
    if (n_ovf == 0) return;
    extern __shared__ __align__(16) uint32_t sm[];
    load_blob_to_smem(blob, blob_words, sm);
    const DevInfoView d = make_view(sm);
    const uint32_t *adj = d.h->adj;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *q = sm + ((blob_words + 3u) & ~3u) + warp * kQueueWords;
    unsigned long long pairs = 0;
    Blocks B;
    B.nb = 0;
    uint32_t cur_idx = kFull;
    for (;;) {
        uint32_t c = 0;
        if (lane == 0) c = atomicAdd(&lc->chunk_next, 1u);
        c = __shfl_sync(kFull, c, 0);
        if (c >= n_chunks) break;
        // largest idx with ovf_off[idx] <= c (ovf_off increases with idx)
        uint32_t lo_i = 0, hi_i = n_ovf - 1;
        while (lo_i < hi_i) {
            uint32_t mid = (lo_i + hi_i + 1) >> 1;
            if (ovf_off[mid] <= c) lo_i = mid;
            else hi_i = mid - 1;
        }
        const uint32_t idx = lo_i;
        const uint32_t S = ovf_set[idx];
        const uint32_t P = ovf_P[idx];
        if (MODE == kModeMpdp && idx != cur_idx) find_blocks(S, adj, B);
        cur_idx = idx;
        const uint32_t W = ovf_work(MODE, P);
        uint32_t lo = (c - ovf_off[idx]) * kChunk;
        uint32_t hi = lo + kChunk < W ? lo + kChunk : W;
        LaneBest best;
        best.init();
        if constexpr (MODE == kModeDpsub) eval_range_dpsub(d, adj, S, P, lo, hi, memo, q, ccc != 0, best);
        else eval_range<MODE>(d, adj, S, B, lo, hi, memo, q, ccc != 0, best);
        unsigned long long mk, fk;
        warp_winner(best, mk, fk);
        if (lane == 0) {
            if (mk != ~0ull) atomicMin(&ovf_key[idx], mk);
            atomicMin(&ovf_first[idx], fk);
        }
        pairs += best.n_valid;
    }
    pairs = __reduce_add_sync(kFull, (uint32_t)pairs);
    if (lane == 0 && pairs) atomicAdd(&glob->evaluated_pairs, pairs);
}

template <int MODE>
__global__ void __launch_bounds__(kBlock) k_ovf_finalize(const uint32_t *__restrict__ blob, uint32_t blob_words,
                                                         LevelCounters *__restrict__ lc, float4 *__restrict__ memo,
                                                         uint32_t *__restrict__ memo_left,
                                                         const uint32_t *__restrict__ ovf_set,
                                                         const unsigned long long *__restrict__ ovf_key,
                                                         const unsigned long long *__restrict__ ovf_first) {
    const uint32_t n_ovf = (uint32_t)(lc->ovf_packed >> 40);
    if (n_ovf == 0) return;
    extern __shared__ __align__(16) uint32_t sm[];
    load_blob_to_smem(blob, blob_words, sm);
    const DevInfoView d = make_view(sm);
    const uint32_t *adj = d.h->adj;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n_ovf; idx += gridDim.x * blockDim.x) {
        const uint32_t S = ovf_set[idx];
        const unsigned long long first = ovf_first[idx];
        const uint32_t p = (first & 1ull) ? (uint32_t)(first >> 1) : (uint32_t)ovf_key[idx];
        uint32_t L, R;
        if (MODE == kModeDpsub || d.h->index_order) {
            L = pdep32(p + 1u, S);
            R = S ^ L;
        } else {
            Blocks B;
            find_blocks(S, adj, B);
            int b = 0;
            while (b + 1 < B.nb && B.prefix[b + 1] <= p) b++;
            uint32_t blk = B.mask[b];
            uint32_t lb = pdep32(p - B.prefix[b] + 1u, blk);
            uint32_t rb = blk ^ lb;
            L = grow(lowest(lb), S & ~rb, adj);
            R = grow(lowest(rb), S & ~lb, adj);
        }
        RelVal l = load_rel(memo, L, d.h->hz_packed), r = load_rel(memo, R, d.h->hz_packed);
        RelVal out = join_eval(d, L, l, R, r);
        memo_write(*d.h, memo, memo_left, S, out, L);
    }
}

// ---------------------------------------------------------------------------
// k_dense: plain DPsub over all subsets of dense graphs with plain classes
// (DevHeader::pairs_plain; a clique of 18 relations has 193 M unordered splits,
// every one valid).  The splits L = pdep(v, S), v = 1 .. 2^(k-1) - 1, and their
// mirrors 2^k - 1 - v are a set's candidates; a lane takes an aligned slice of
// them, so that the same relations change sides in all lanes at the same time,
// and carries the matching classes from split to split (pairs_flip: two
// relations change sides on average) instead of gathering the class rows of
// all relations; nearly every split is valid, so none is queued.
// Bound: issue (54 to 67 % of the slots), 390 to 460 instructions a split, 160 of
// them the selectivity product in class order over the 66 classes of a set of 12
// relations of the clique.  The 18-relation clique takes 3.7 ms; with the class
// rows as they are and a search for each lane's matching classes it took 8.1,
// and with 4 blocks an SM (64 registers, some spilled) 3.9.  share: values of v per warp, a power
// of two; a set of at most that many is one warp's and written at once,
// otherwise the shares fold their keys (as k_ovf_chunks does) and the warp of a
// set's last share writes the winner.
// ---------------------------------------------------------------------------
constexpr uint32_t kDenseWhole = 1024u;   // an 11-relation set

// plain DPsub keeps the all-subsets enumeration on graphs with at least half
// of all possible edges (apply_dpsub_csg); sparse ones only come here with
// gpuqo_dpsub_csg_enable off, and their invalid subsets are better queued
static bool dense_pairs(const DevHeader &h) {
    uint64_t degrees = 0;
    for (int i = 0; i < h.n; i++) degrees += (uint64_t)__builtin_popcount(h.adj[i]);
    return h.pairs_plain != 0u && 2 * degrees >= (uint64_t)h.n * (uint64_t)(h.n - 1);
}

template <int NW>
__global__ void __launch_bounds__(kBlock, 3) k_dense(const uint32_t *__restrict__ blob, uint32_t blob_words, int k,
                                                     const uint32_t *__restrict__ sets, LevelCounters *__restrict__ lc,
                                                     float4 *__restrict__ memo, uint32_t *__restrict__ memo_left,
                                                     unsigned long long *__restrict__ keys,
                                                     unsigned long long *__restrict__ firsts,
                                                     uint32_t *__restrict__ parts,
                                                     GlobalCounters *__restrict__ glob, uint32_t share) {
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ PairTable<NW> tabs[kWarpsPerBlock];
    load_blob_to_smem(blob, blob_words, sm);
    const DevInfoView d = make_view(sm);
    const DevHeader &h = *d.h;
    const uint32_t *adj = h.adj;
    const PlainParams pp = plain_params(h);
    const uint32_t lane = threadIdx.x & 31u;
    PairTable<NW> &tab = tabs[threadIdx.x >> 5];
    const uint32_t count = lc->n_sets, V = 1u << (k - 1), P = 2u * V - 2u;
    const uint32_t per_set = V / share, per = (share + 31u) / 32u;
    const unsigned long long items = (unsigned long long)count * per_set;
    uint32_t found = 0u;
    for (unsigned long long item = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); item < items;
         item += gridDim.x * kWarpsPerBlock) {
        const uint32_t idx = (uint32_t)(item / per_set), part = (uint32_t)(item % per_set);
        const uint32_t S = sets[idx];
        const int classes = pairs_table<NW>(d, S, lane, tab);
        uint32_t odd[4 * NW];
#pragma unroll
        for (int w = 0; w < 4 * NW; w++) odd[w] = 0u;
        uint32_t v = part * share + per * lane;
        const uint32_t end = per * lane < share ? v + per : v;
        uint32_t L = v < end ? pdep32(v, S) : 0u;
        pairs_flip<NW>(tab, L, odd);
        // all relations of S joined pairwise: every split is valid
        const bool whole_clique = __all_sync(kFull, !((S >> lane) & 1u) || (adj[lane] & S) == (S ^ (1u << lane)));
        // The first minimum in the order of the candidates: splits come in that
        // order, mirrors in reverse and after every split, so that a cost equal
        // to a mirror's takes its place and one equal to a split's does not.
        float best = INFINITY, rows = 0.0f, startup = 0.0f;
        uint32_t best_v = 0u;
        bool of_mirror = true;
        uint32_t first = kFull;
        bool first_nan = false;
        int width = 0;
        float4 l = __ldcg(memo + L), r = __ldcg(memo + (S ^ L));
        for (; v < end; v++) {
            // the next split's entries are on their way while this one is
            // costed (whatever they hold, if it is not valid)
            const uint32_t next = next_subset(L, S);
            const float4 l_next = __ldcg(memo + next), r_next = __ldcg(memo + (S ^ next));
            if (whole_clique ? L != 0u : (is_connected(L, adj) && is_connected(S ^ L, adj))) {
                JoinCost lr, rl;
                pairs_mirror<NW>(d, pp, tab, classes, odd, l, r, lr, rl);
                width = (int)((__float_as_uint(l.w) & kWidthMask) + (__float_as_uint(r.w) & kWidthMask));
                found += 2u;
                // the lane's first valid candidate is its first valid split as
                // it stands: mirrors come after every split
                if (first == kFull) {
                    first = v - 1u;
                    first_nan = isnan(lr.total);
                }
                if (of_mirror ? lr.total <= best : lr.total < best) {
                    best = lr.total;
                    rows = lr.rows;
                    startup = lr.startup;
                    best_v = v;
                    of_mirror = false;
                }
                if (of_mirror ? rl.total <= best : rl.total < best) {
                    best = rl.total;
                    rows = rl.rows;
                    startup = rl.startup;
                    best_v = v;
                    of_mirror = true;
                }
            }
            pairs_flip<NW>(tab, L ^ next, odd);
            L = next;
            l = l_next;
            r = r_next;
        }
        __syncwarp();
        const uint32_t kh = best_v ? ord_float(best) : kFull;
        const uint32_t kl = best_v ? (of_mirror ? P - best_v : best_v - 1u) : kFull;
        const uint32_t mh = __reduce_min_sync(kFull, kh);
        const uint32_t ml = __reduce_min_sync(kFull, kh == mh ? kl : kFull);
        const uint32_t mf = __reduce_min_sync(kFull, first);
        const bool nan = __any_sync(kFull, first == mf && first_nan);
        unsigned long long win = nan ? mf : ml;
        if (per_set > 1u) {
            uint32_t last = 0u;
            if (lane == 0u) {
                const unsigned long long mk = ((unsigned long long)mh << 32) | ml;
                if (mk != ~0ull) atomicMin(keys + idx, mk);
                atomicMin(firsts + idx, ((unsigned long long)mf << 1) | (nan ? 1ull : 0ull));
                __threadfence();
                if (atomicAdd(parts + idx, 1u) == per_set - 1u) {
                    __threadfence();
                    const unsigned long long f = __ldcg(firsts + idx);
                    win = (f & 1ull) ? f >> 1 : __ldcg(keys + idx) & 0xFFFFFFFFull;
                    last = 1u;
                    keys[idx] = firsts[idx] = ~0ull;   // as the next level expects them
                    parts[idx] = 0u;
                }
            }
            if (!__shfl_sync(kFull, last, 0)) continue;
            win = __shfl_sync(kFull, win, 0);
        } else if (!nan) {
            if (kh == mh && kl == ml && best_v != 0u) {
                RelVal out;
                out.rows = rows;
                out.startup = startup;
                out.total = best;
                out.width = width;
                memo_write(h, memo, memo_left, S, out, pdep32(ml + 1u, S));
            }
            continue;
        }
        // the winning candidate of shares, or a NaN found first, once more
        L = pdep32((uint32_t)win + 1u, S);
#pragma unroll
        for (int w = 0; w < 4 * NW; w++) odd[w] = 0u;
        pairs_flip<NW>(tab, L, odd);
        l = __ldcg(memo + L);
        r = __ldcg(memo + (S ^ L));
        JoinCost lr, rl;
        pairs_mirror<NW>(d, pp, tab, classes, odd, l, r, lr, rl);
        if (lane == 0u) {
            RelVal out;
            out.rows = lr.rows;
            out.startup = lr.startup;
            out.total = lr.total;
            out.width = (int)((__float_as_uint(l.w) & kWidthMask) + (__float_as_uint(r.w) & kWidthMask));
            memo_write(h, memo, memo_left, S, out, L);
        }
    }
    found = __reduce_add_sync(kFull, found);
    if (lane == 0u && found) atomicAdd(&glob->evaluated_pairs, (unsigned long long)found);
}

// ---------------------------------------------------------------------------
// DPsize (gpuqo_cpu_dpsize.cu:28-96 with gpuqo_cpu_sequential.cu:28-58): for
// join size k = 2..n, left size m = k-1 down to 1, every relation set L of the
// level-m list and R of the level-(k-m) list, in list order, a disjoint and
// connected pair (L, R) is costed as L joining R; the set L + R keeps its
// first strict minimum (a NaN cost first found is kept), and is appended to
// the level-k list when it is first produced.  The level-1 list is the
// iteration order of the reference's unordered_map memo after the base
// relations are inserted (dpsize_level1_places); later lists are in
// discovery order.
//
// Here every connected k-set S is costed on its own (one warp, the valid
// splits of S from the biconnected-block enumeration), with each split keyed
// by its place in that loop: G = off[|L|] + pos[L], off[m] = the sizes of
// levels m+1 .. k-1 (larger left sides first), pos[] the position of a set in
// its level list.  The lexicographic minimum of (cost, G) is the reference's
// first strict minimum.  S is first produced by its split of smallest
// (G, pos[R]); that split always has |L| = k-1 (every connected set has a
// relation whose removal leaves it connected), so S's discovery key is
// (pos[L*], pos[v*]) with v* the relation outside L*.  The level-k list order
// follows from the keys without a sort: the sets discovered from one L* are
// L* + v for different relations v, so one 32-bit mask per level-(k-1) set
// collects the pos[v] of its discoveries, an exclusive scan of the mask
// popcounts gives each L*'s first place, and a set's place is that plus the
// number of lower bits in its L*'s mask.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) k_dpsize_eval(const uint32_t *__restrict__ blob, uint32_t blob_words,
                                                        int k, const uint32_t *__restrict__ sets,
                                                        const LevelCounters *__restrict__ lvl,
                                                        float4 *__restrict__ memo, uint32_t *__restrict__ memo_left,
                                                        const uint32_t *__restrict__ pos,
                                                        unsigned long long *__restrict__ disc,
                                                        uint32_t *__restrict__ bmask,
                                                        GlobalCounters *__restrict__ glob) {
    const uint32_t count = __ldcg(&lvl[k].n_sets);
    if (count == 0u) return;
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ uint32_t off[33];
    load_blob_to_smem(blob, blob_words, sm);
    const DevInfoView d = make_view(sm);
    const uint32_t *adj = d.h->adj;
    if (threadIdx.x == 0) {
        // off[m] = sizes of the levels m+1 .. k-1; level 1 holds the n relations
        uint32_t acc = 0u;
        for (int m = k - 1; m >= 1; m--) {
            off[m] = acc;
            acc += (m == 1) ? (uint32_t)d.h->n : __ldcg(&lvl[m].n_sets);
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
    unsigned long long pairs = 0;
    Blocks B;
    CycleCache cc;
    for (uint32_t i = blockIdx.x * kWarpsPerBlock + warp; i < count; i += nwarps) {
        const uint32_t S = __ldcg(sets + i);
        find_blocks(S, adj, B);
        const uint32_t P = B.etotal;
        LaneBest best;
        best.init();
        unsigned long long dmin = ~0ull;
        int b = 0;
        for (uint32_t c = (uint32_t)lane; c < P; c += 32u) {
            uint32_t L, R, key;
            if (!mpdp_candidate(S, B, adj, c, b, L, R, key, cc)) continue;
            const uint32_t g = off[__popc(L)] + __ldcg(pos + L);
            const unsigned long long dk = ((unsigned long long)g << 32) | __ldcg(pos + R);
            if (dk < dmin) dmin = dk;
            const RelVal l = load_rel(memo, L, d.h->hz_packed), r = load_rel(memo, R, d.h->hz_packed);
            best_update(best, g, L, join_eval(d, L, l, R, r));
        }
        unsigned long long mk, fk;
        const WarpWinner w = warp_winner(best, mk, fk);
        if (w.is_writer) {
            if (w.use_nan) memo_write(*d.h, memo, memo_left, S, best.nan_val, best.nan_left);
            else memo_write(*d.h, memo, memo_left, S, best.val, best.left);
        }
        const uint32_t dh = __reduce_min_sync(kFull, (uint32_t)(dmin >> 32));
        const uint32_t dl = __reduce_min_sync(kFull, (uint32_t)(dmin >> 32) == dh ? (uint32_t)dmin : kFull);
        if (lane == 0) {
            disc[i] = ((unsigned long long)dh << 32) | dl;
            atomicOr(bmask + dh, 1u << dl);
        }
        pairs += best.n_valid;
    }
    pairs = __reduce_add_sync(kFull, (uint32_t)pairs);
    if (lane == 0 && pairs) atomicAdd(&glob->evaluated_pairs, pairs);
}

constexpr uint32_t kScanTile = kBlock * 4;   // mask words per block of the place scan

// block b: the popcount total of bmask[b * kScanTile ..) (entries < level k-1's size)
__global__ void __launch_bounds__(kBlock) k_dpsize_scan_tiles(const uint32_t *__restrict__ bmask,
                                                              const LevelCounters *__restrict__ lvl, int km1, int n,
                                                              uint32_t *__restrict__ tile_sum) {
    const uint32_t cnt = km1 == 1 ? (uint32_t)n : __ldcg(&lvl[km1].n_sets);
    const uint32_t base = blockIdx.x * kScanTile;
    if (base >= cnt) return;
    uint32_t v = 0u;
    for (uint32_t j = threadIdx.x; j < kScanTile; j += kBlock)
        if (base + j < cnt) v += (uint32_t)__popc(__ldcg(bmask + base + j));
    v = __reduce_add_sync(kFull, v);
    __shared__ uint32_t ws[kWarpsPerBlock];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0u;
        for (int w = 0; w < kWarpsPerBlock; w++) t += ws[w];
        tile_sum[blockIdx.x] = t;
    }
}

// one block: exclusive scan of the tile totals, in place
__global__ void __launch_bounds__(kBlock) k_dpsize_scan_top(uint32_t *__restrict__ tile_sum,
                                                            const LevelCounters *__restrict__ lvl, int km1, int n) {
    const uint32_t cnt = km1 == 1 ? (uint32_t)n : __ldcg(&lvl[km1].n_sets);
    const uint32_t tiles = (cnt + kScanTile - 1u) / kScanTile;
    __shared__ uint32_t carry;
    __shared__ uint32_t ws[kWarpsPerBlock];
    if (threadIdx.x == 0) carry = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t base = 0; base < tiles; base += kBlock) {
        const uint32_t idx = base + threadIdx.x;
        const uint32_t v = idx < tiles ? tile_sum[idx] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) ws[warp] = incl;
        __syncthreads();
        uint32_t wpre = 0u, total = 0u;
        for (int w = 0; w < kWarpsPerBlock; w++) {
            if (w < warp) wpre += ws[w];
            total += ws[w];
        }
        if (idx < tiles) tile_sum[idx] = carry + wpre + incl - v;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
}

// block b: bstart[j] = exclusive prefix of the mask popcounts for the masks j
// of tile b (the tile's offset from k_dpsize_scan_top plus the popcounts of
// the tile's earlier masks); each thread takes 4 consecutive masks
__global__ void __launch_bounds__(kBlock) k_dpsize_scan_fill(const uint32_t *__restrict__ bmask,
                                                             const LevelCounters *__restrict__ lvl, int km1, int n,
                                                             const uint32_t *__restrict__ tile_sum,
                                                             uint32_t *__restrict__ bstart) {
    const uint32_t cnt = km1 == 1 ? (uint32_t)n : __ldcg(&lvl[km1].n_sets);
    const uint32_t base = blockIdx.x * kScanTile;
    if (base >= cnt) return;
    const uint32_t j0 = base + threadIdx.x * 4u;
    uint32_t c[4], tot = 0u;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        c[q] = (j0 + q < cnt) ? (uint32_t)__popc(__ldcg(bmask + j0 + q)) : 0u;
        tot += c[q];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    __shared__ uint32_t ws[kWarpsPerBlock];
    if (lane == 31) ws[warp] = incl;
    __syncthreads();
    uint32_t run = __ldcg(tile_sum + blockIdx.x) + incl - tot;
    for (int w = 0; w < warp; w++) run += ws[w];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (j0 + q < cnt) bstart[j0 + q] = run;
        run += c[q];
    }
}

// every set of level k: its place in the level-k list
__global__ void __launch_bounds__(kBlock) k_dpsize_place(const uint32_t *__restrict__ sets,
                                                         const LevelCounters *__restrict__ lvl, int k,
                                                         const unsigned long long *__restrict__ disc,
                                                         const uint32_t *__restrict__ bmask,
                                                         const uint32_t *__restrict__ bstart,
                                                         uint32_t *__restrict__ pos) {
    const uint32_t count = __ldcg(&lvl[k].n_sets);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const unsigned long long dk = __ldcg(disc + i);
        const uint32_t bl = (uint32_t)(dk >> 32), v = (uint32_t)dk;
        pos[__ldcg(sets + i)] = __ldcg(bstart + bl) + (uint32_t)__popc(__ldcg(bmask + bl) & ((1u << v) - 1u));
    }
}

// the masks of the level-(k-1) sets, cleared once every place is read
__global__ void __launch_bounds__(kBlock) k_dpsize_clear(uint32_t *__restrict__ bmask,
                                                         const LevelCounters *__restrict__ lvl, int km1, int n) {
    const uint32_t cnt = km1 == 1 ? (uint32_t)n : __ldcg(&lvl[km1].n_sets);
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x) bmask[j] = 0u;
}

// the level-1 list: pos[1 << i] = place of relation i
__global__ void k_dpsize_init(uint32_t *__restrict__ pos, const uint32_t *__restrict__ level1, int n) {
    const int i = threadIdx.x;
    if (i < n) pos[1u << i] = level1[i];
}

// ---------------------------------------------------------------------------
// base relations and plan extraction
// ---------------------------------------------------------------------------
__global__ void k_init_base(const uint32_t *__restrict__ blob, float4 *__restrict__ memo,
                            uint32_t *__restrict__ memo_left) {
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob);
    int i = threadIdx.x;
    if (i < h->n) {
        // gpuqo_cpu_sequential.cu:80-92: base relation memo entries
        memo[1u << i] = base_entry(*h, i);
        memo_left[1u << i] = 0u;
    }
}

__global__ void k_extract(const float4 *__restrict__ memo, const uint32_t *__restrict__ memo_left, uint32_t full,
                          const uint32_t *__restrict__ blob, TreeNode *__restrict__ out, int *__restrict__ n_out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const uint32_t wmask = reinterpret_cast<const DevHeader *>(blob)->hz_packed ? kWidthMask : 0xFFFFFFFFu;
    // iterative preorder walk; node i's children are appended after it
    int n = 0;
    uint32_t stack_set[64];
    int stack_parent[64];
    int stack_side[64];
    int sp = 0;
    stack_set[sp] = full;
    stack_parent[sp] = -1;
    stack_side[sp] = 0;
    sp++;
    while (sp > 0 && n < 64) {
        sp--;
        uint32_t s = stack_set[sp];
        int parent = stack_parent[sp], side = stack_side[sp];
        float4 v = memo[s];
        TreeNode t;
        t.set = s;
        t.left = -1;
        t.right = -1;
        t.rows = v.x;
        t.startup = v.y;
        t.total = v.z;
        t.width = (int)(__float_as_uint(v.w) & wmask);
        int me = n++;
        out[me] = t;
        if (parent >= 0) {
            if (side == 0) out[parent].left = me;
            else out[parent].right = me;
        }
        uint32_t l = memo_left[s] & s;
        if (__popc(s) > 1 && l != 0u && l != s && sp + 2 <= 64) {
            uint32_t r = s ^ l;
            stack_set[sp] = r;
            stack_parent[sp] = me;
            stack_side[sp] = 1;
            sp++;
            stack_set[sp] = l;
            stack_parent[sp] = me;
            stack_side[sp] = 0;
            sp++;
        }
    }
    *n_out = n;
}

// ---------------------------------------------------------------------------
// host engine
// ---------------------------------------------------------------------------
static uint64_t binom64(int n, int k) {
    if (k < 0 || k > n) return 0;
    uint64_t r = 1;
    for (int i = 1; i <= k; i++) r = r * (uint64_t)(n - k + i) / (uint64_t)i;
    return r;
}

static uint64_t max_level_sets(int n) {
    uint64_t m = 1;
    for (int k = 0; k <= n; k++) m = std::max(m, binom64(n, k));
    return m;
}

uint64_t engine_bytes_needed(int n) {
    uint64_t memo = (1ull << n) * (sizeof(float4) + sizeof(uint32_t));
    uint64_t lv = max_level_sets(n) * (4ull * 4 + 8ull * 2);
    return memo + lv + (1u << 20);
}

// a failed allocation is GPUQO_B200_ERR_NOMEM (it leaves no sticky error:
// the next call may succeed), any other failure GPUQO_B200_ERR_CUDA
#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            err = std::string(#call) + ": " + cudaGetErrorString(e_);                     \
            cudaGetLastError();   /* reported here: not by the next call's check too */   \
            return e_ == cudaErrorMemoryAllocation ? GPUQO_B200_ERR_NOMEM : GPUQO_B200_ERR_CUDA; \
        }                                                                                 \
    } while (0)

// gpuqo_b200_device_memory_mb: when > 0, a DP whose arena would need more
// device memory than this is refused with GPUQO_B200_ERR_NOMEM before any
// allocation (the engines keep what they hold, so later calls are unaffected)
// A buffer's pointer is null from the moment it is freed, so that an
// allocation that fails leaves nothing a later call could use or free again.
template <class T> static void release(T *&p) {
    if (p) cudaFree(p);
    p = nullptr;
}

static int over_budget(uint64_t bytes, const char *what, std::string &err) {
    const int mb = gpuqo_b200_device_memory_mb;
    if (mb <= 0 || bytes <= ((uint64_t)mb << 20)) return 0;
    err = std::string(what) + " needs " + std::to_string(bytes >> 20) + " MB of device memory; " +
          "gpuqo_b200_device_memory_mb allows " + std::to_string(mb);
    return GPUQO_B200_ERR_NOMEM;
}

struct GraphKey {
    int n, mode, ccc, profile;
    bool operator<(const GraphKey &o) const {
        if (n != o.n) return n < o.n;
        if (mode != o.mode) return mode < o.mode;
        if (ccc != o.ccc) return ccc < o.ccc;
        return profile < o.profile;
    }
};

// Parameters the autotuner (engine_autotune) measures; these defaults apply
// until it runs.  Neither changes a plan, only which kernel variant runs.
struct Tuning {
    // tree queries with up to this many connected sets per level run
    // k_dp_tree<2>, those with more than single_wide_level_sets k_dp_tree<4>
    // (device time of the 2- / 3- / 4-blocks variant: star-18, 7 k sets per
    // level, 95 / 103 / 120 us; star-20, 26 k, 159 / 156 / 176; star-22, 95 k,
    // 381 / 372 / 384; star-24, 350 k, 1357 / 1210 / 1194; star-26, 1.3 M,
    // 6182 / 5363 / 5591; star-27, 2.5 M, 13.5 / 11.8 / 12.6 ms; snowflake-28,
    // 12 k, 217 / 227 / 268 us; snowflake-30, 39 k, 427 / 430 / 474: the third
    // one wins by 1 % between 350 and 700 k, which is left to the autotuner)
    double single_narrow_level_sets = 16384.0;
    double single_wide_level_sets = 1e30;
    double batch_single_sets = double(1u << 20);   // a batch hands larger tree queries to k_dp_tree
    bool tuned = false;
};
constexpr int kMaxDevices = 64;
static Tuning g_tuning[kMaxDevices];            // per device, guarded by g_dev_mu

static double tree_connected_sets(const DevHeader *h);

// Connected sets of a tree-shaped query graph by size (count[k], k = 1..n; at
// most C(30, 15) each): with g_v(x) counting the connected sets whose relation
// nearest to relation 0 is v, g_v = x * prod over v's children c of
// (1 + g_c), O(n^2) steps in all.  Returns their total.
static double tree_level_counts(const DevHeader *h, uint32_t (&count)[33]) {
    const int n = h->n;
    int order[32], parent[32], size[32], m = 0;
    uint32_t g[32][33];
    uint32_t seen = 1u;
    order[m++] = 0;
    parent[0] = -1;
    for (int i = 0; i < m; i++) {
        uint32_t nb = h->adj[order[i]] & ~seen;
        seen |= nb;
        for (; nb; nb &= nb - 1u) {
            const int c = __builtin_ctz(nb);
            parent[c] = order[i];
            order[m++] = c;
        }
    }
    for (int v = 0; v < n; v++) {
        size[v] = 1;
        g[v][0] = 0u;
        g[v][1] = 1u;
    }
    for (int k = 0; k <= 32; k++) count[k] = 0u;
    double total = 0.0;
    for (int i = m - 1; i >= 0; i--) {
        const int v = order[i], p = parent[v];
        for (int k = 1; k <= size[v]; k++) {
            count[k] += g[v][k];
            total += (double)g[v][k];
        }
        if (p < 0) continue;
        uint32_t nx[33] = {};
        for (int a = 1; a <= size[p]; a++) {
            nx[a] += g[p][a];
            for (int b = 1; b <= size[v]; b++) nx[a + b] += g[p][a] * g[v][b];
        }
        size[p] += size[v];
        for (int k = 1; k <= size[p]; k++) g[p][k] = nx[k];
    }
    return total;
}

// The order in which the tree kernels list connected sets (tree_extension_mask)
// for a memo of `slots` entries of which `sets` are used, a sector of 32 bytes
// each: near once the sectors exceed the L2 cache, or, for plain trees, whose
// cost does not cover the misses, once the memo's span exceeds 512 MB, some 256
// pages of 2 MB (snowflake-25, 512 MB: 156 us by the largest leaf, 158 near;
// snowflake-26: 191 and 178; -30: 732 and 453; star-22, 67 MB of sectors: 394 and
// 391, star-24: 1438 and 1242, star-26 / 27 / 28: 11.6 / 26.4 / 57.3 ms and 5.4 /
// 11.7 / 25.5; with statistics snowflake-28 454 and 460 us).
static bool near_order(uint64_t slots, double sets, int layout, int l2_bytes) {
    return 32.0 * sets > (double)l2_bytes || (layout == kTreePlain && 16ull * slots > (512ull << 20));
}

// cpu_dpsize's level-1 list (gpuqo_cpu_dpsize.cu:43-48 after
// gpuqo_cpu_sequential.cu:73-84): the iteration order of its unordered_map
// memo once base relation i (key 2^(i+1), whose hash is the key itself) has
// been inserted for i = 0 .. n-1.  The same standard-library container,
// filled the same way, gives the same order; place[i] = position of relation i.
static std::vector<uint32_t> dpsize_level1_places(int n) {
    std::unordered_map<uint32_t, int> m;
    for (int i = 0; i < n; i++) m.insert(std::make_pair(1u << (i + 1), i));
    std::vector<uint32_t> place((size_t)n, 0u);
    uint32_t p = 0;
    for (const auto &kv : m) place[(size_t)kv.second] = p++;
    return place;
}

// Per-run control words of the single-query engine, contiguous so that one
// memset clears the counters and one copy brings everything back.
struct EngineCtl {
    LevelCounters lvl[33];
    GlobalCounters glob;
    unsigned bar[4];                   // grid barrier of k_dp_tree: arrivals, -, error flag
    int tree_n;
    int pad;
    TreeNode tree[64];
};
constexpr size_t kCtlClearBytes = offsetof(EngineCtl, pad);   // lvl .. tree_n

// largest cluster of k_dp_tree (the portable size), and the blocks' worth of
// splits of the widest level up to which a cluster runs the query
constexpr int kTreeCluster = 8;
constexpr int kTreeClusterLevel = 16;

// one cluster of `blocks` blocks
static cudaError_t launch_cluster(const void *fn, int blocks, size_t smem, void **args, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kBlock);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)blocks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

class Engine {
public:
    int device = -1;
    int sm_count = 148, l2_bytes = 0;
    cudaStream_t stream = nullptr;
    DevArena a;
    int cap_n = -1;                    // arena sized for this many relations
    uint64_t cap_sets = 0;
    uint32_t blob_cap_words = 0;
    uint32_t *h_blob = nullptr;        // pinned staging
    uint32_t h_level1[32];             // staging of the DPsize level-1 list (copied before each launch)
    EngineCtl *d_ctl = nullptr;        // device control words (a.lvl, a.glob, a.bar, a.tree_n, a.tree point here)
    EngineCtl *h_ctl = nullptr;        // pinned copy
    TreeNode *h_tree = nullptr;        // views into h_ctl
    int *h_tree_n = nullptr;
    GlobalCounters *h_glob = nullptr;
    LevelCounters *h_lvl = nullptr;
    std::map<GraphKey, cudaGraphExec_t> graphs;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::vector<cudaEvent_t> kev;      // per-level eval events (profile mode)
    int n_kernels = 0;                 // kernels per DP run
    // k_dp_tree leaves its counters at zero and the barrier's arrivals where
    // the next launch goes on: whether they are so, and the arrivals
    bool ctl_clean = false;
    unsigned bar_base = 0, bar_after = 0;
    double plan_sets = 0.0;            // connected sets and pairs of the last persistent run
    uint64_t plan_pairs = 0;
    std::map<size_t, int> coop_blocks; // (dynamic shared bytes, variant) -> co-resident blocks of k_dp_tree (0: none)
    std::map<const void *, size_t> smem_limit;   // dynamic shared memory that its variants are allowed
    int force_minb = 0;                // autotuner: run this k_dp_tree variant (2, 3 or 4); 0 = by the tuning record
    bool coop_off = false;             // cooperative launch refused on this device
    bool barrier_timed_out = false;    // a grid barrier of k_dp_tree gave up: per-level launches until reset
    std::map<GraphKey, int> graph_kernels;
    float *flush = nullptr;            // L2 flush buffer (timing only)
    bool ready = false;                // init has come to its end

    int init(std::string &err) {
        if (ready) return 0;
        CK(cudaGetDevice(&device));
        CK(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
        CK(cudaDeviceGetAttribute(&l2_bytes, cudaDevAttrL2CacheSize, device));
        if (!stream) CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        if (!ev0) CK(cudaEventCreate(&ev0));
        if (!ev1) CK(cudaEventCreate(&ev1));
        kev.resize(2 * 34);
        for (auto &e : kev)
            if (!e) CK(cudaEventCreate(&e));
        if (!d_ctl) CK(cudaMalloc(&d_ctl, sizeof(EngineCtl)));
        if (!h_ctl) CK(cudaMallocHost(&h_ctl, sizeof(EngineCtl)));
        a.lvl = d_ctl->lvl;
        a.glob = &d_ctl->glob;
        a.bar = d_ctl->bar;
        a.tree_n = &d_ctl->tree_n;
        a.tree = d_ctl->tree;
        h_lvl = h_ctl->lvl;
        h_glob = &h_ctl->glob;
        h_tree_n = &h_ctl->tree_n;
        h_tree = h_ctl->tree;
        if (!a.binom) CK(cudaMalloc(&a.binom, 33 * 33 * sizeof(uint32_t)));
        std::vector<uint32_t> bt(33 * 33, 0);
        for (int i = 0; i <= 32; i++)
            for (int j = 0; j <= 32; j++) {
                uint64_t v = binom64(i, j);
                bt[i * 33 + j] = v > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)v;
            }
        CK(cudaMemcpy(a.binom, bt.data(), bt.size() * 4, cudaMemcpyHostToDevice));
        ready = true;
        return 0;
    }

    void drop_graphs() {
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second);
        graphs.clear();
    }

    int ensure(int n, uint32_t blob_words, std::string &err) {
        if (blob_words > blob_cap_words) {
            drop_graphs();
            blob_cap_words = 0;
            release(a.blob);
            if (h_blob) cudaFreeHost(h_blob);
            h_blob = nullptr;
            uint32_t cap = std::max<uint32_t>((blob_words + 511u) & ~511u, 16384u);
            CK(cudaMalloc(&a.blob, cap * 4));
            CK(cudaMallocHost(&h_blob, cap * 4));
            blob_cap_words = cap;
        }
        // the budget bounds what one DP needs, whatever the engine already holds
        if (int rc = over_budget(engine_bytes_needed(n), "the exact DP's dense memo and level lists", err)) return rc;
        if (n <= cap_n) return 0;
        drop_graphs();
        cap_n = -1;
        release(a.memo);
        release(a.memo_left);
        release(a.sets);
        release(a.sets2);
        release(a.seen);
        release(a.ovf_set);
        release(a.ovf_P);
        release(a.ovf_off);
        release(a.ovf_key);
        release(a.ovf_first);
        uint64_t slots = 1ull << n;
        uint64_t ms = max_level_sets(n);
        CK(cudaMalloc(&a.memo, slots * sizeof(float4)));
        CK(cudaMalloc(&a.memo_left, slots * sizeof(uint32_t)));
        CK(cudaMalloc(&a.sets, ms * sizeof(uint32_t)));
        CK(cudaMalloc(&a.sets2, ms * sizeof(uint32_t)));
        CK(cudaMalloc(&a.seen, std::max<uint64_t>(slots / 8, 4)));
        CK(cudaMalloc(&a.ovf_set, ms * sizeof(uint32_t)));
        CK(cudaMalloc(&a.ovf_P, ms * sizeof(uint32_t)));
        CK(cudaMalloc(&a.ovf_off, ms * sizeof(uint32_t)));
        CK(cudaMalloc(&a.ovf_key, ms * sizeof(unsigned long long)));
        CK(cudaMalloc(&a.ovf_first, ms * sizeof(unsigned long long)));
        cap_n = n;
        cap_sets = ms;
        return 0;
    }

    int dpsize_cap_n = -1;             // DPsize buffers sized for this many relations

    int ensure_dpsize(int n, std::string &err) {
        const uint64_t ms = max_level_sets(n);
        const uint64_t tiles = ms / kScanTile + 2;
        if (int rc = over_budget(engine_bytes_needed(n) + (1ull << n) * 4 + ms * 16 + tiles * 4,
                                 "DPsize's dense memo, level lists and place arrays", err))
            return rc;
        if (n <= dpsize_cap_n) return 0;
        drop_graphs();
        dpsize_cap_n = -1;
        release(a.pos);
        release(a.bmask);
        release(a.bstart);
        release(a.tile_sum);
        release(a.disc);
        CK(cudaMalloc(&a.pos, (1ull << n) * sizeof(uint32_t)));
        CK(cudaMalloc(&a.bmask, ms * sizeof(uint32_t)));
        CK(cudaMalloc(&a.bstart, ms * sizeof(uint32_t)));
        CK(cudaMalloc(&a.tile_sum, tiles * sizeof(uint32_t)));
        CK(cudaMalloc(&a.disc, ms * sizeof(unsigned long long)));
        if (!a.level1) CK(cudaMalloc(&a.level1, 32 * sizeof(uint32_t)));
        dpsize_cap_n = n;
        return 0;
    }

    // DPsize of n relations on `stream` (see k_dpsize_eval)
    int enqueue_dpsize(int n, uint32_t blob_words, std::string &err) {
        const size_t smem = eval_smem(blob_words);
        CK(cudaMemsetAsync(d_ctl, 0, kCtlClearBytes, stream));
        CK(cudaMemsetAsync(a.seen, 0, std::max<uint64_t>((1ull << n) / 8, 4), stream));
        CK(cudaMemsetAsync(a.bmask, 0, max_level_sets(n) * sizeof(uint32_t), stream));
        n_kernels = 0;
        k_init_base<<<1, 32, 0, stream>>>(a.blob, a.memo, a.memo_left);
        k_dpsize_init<<<1, 32, 0, stream>>>(a.pos, a.level1, n);
        n_kernels += 2;
        for (int k = 2; k <= n; k++) {
            const uint64_t total = binom64(n, k);
            uint64_t threads = std::min<uint64_t>((uint64_t)sm_count * 8 * kBlock, (total + 3) / 4);
            threads = std::max<uint64_t>(threads, 32);
            const uint32_t per_thread = (uint32_t)((total + threads - 1) / threads);
            const uint32_t fblocks =
                (uint32_t)((total + (uint64_t)per_thread * kBlock - 1) / ((uint64_t)per_thread * kBlock));
            uint32_t *cur_sets = (k & 1) ? a.sets2 : a.sets;
            const uint32_t *prev_sets = (k & 1) ? a.sets : a.sets2;
            k_level_sets<<<fblocks, kBlock, 0, stream>>>(a.blob, a.binom, n, k, total, per_thread, prev_sets,
                                                         a.lvl + (k - 1), a.seen, cur_sets, a.lvl + k);
            const int eblocks =
                (int)std::min<uint64_t>((uint64_t)sm_count * 4, (total + kWarpsPerBlock - 1) / kWarpsPerBlock);
            CK(cudaEventRecordWithFlags(kev[2 * k], stream, cudaEventRecordExternal));
            k_dpsize_eval<<<eblocks, kBlock, smem, stream>>>(a.blob, blob_words, k, cur_sets, a.lvl, a.memo,
                                                             a.memo_left, a.pos, a.disc, a.bmask, a.glob);
            CK(cudaEventRecordWithFlags(kev[2 * k + 1], stream, cudaEventRecordExternal));
            // places of the level-k sets from the masks of the level-(k-1) sets
            const uint64_t prev_total = binom64(n, k - 1);
            const uint32_t tiles = (uint32_t)((prev_total + kScanTile - 1) / kScanTile);
            k_dpsize_scan_tiles<<<tiles, kBlock, 0, stream>>>(a.bmask, a.lvl, k - 1, n, a.tile_sum);
            k_dpsize_scan_top<<<1, kBlock, 0, stream>>>(a.tile_sum, a.lvl, k - 1, n);
            k_dpsize_scan_fill<<<tiles, kBlock, 0, stream>>>(a.bmask, a.lvl, k - 1, n, a.tile_sum, a.bstart);
            const uint32_t pblocks = (uint32_t)std::min<uint64_t>((uint64_t)sm_count * 8, (total + kBlock - 1) / kBlock);
            k_dpsize_place<<<pblocks, kBlock, 0, stream>>>(cur_sets, a.lvl, k, a.disc, a.bmask, a.bstart, a.pos);
            const uint32_t cblocks =
                (uint32_t)std::min<uint64_t>((uint64_t)sm_count * 8, (prev_total + kBlock - 1) / kBlock);
            k_dpsize_clear<<<cblocks, kBlock, 0, stream>>>(a.bmask, a.lvl, k - 1, n);
            n_kernels += 7;
        }
        const uint32_t full = (n == 32) ? 0xFFFFFFFFu : ((1u << n) - 1u);
        k_extract<<<1, 32, 0, stream>>>(a.memo, a.memo_left, full, a.blob, a.tree, a.tree_n);
        n_kernels++;
        return 0;
    }

    size_t eval_smem(uint32_t blob_words) const {
        return (size_t)(((blob_words + 3u) & ~3u) + kWarpsPerBlock * kQueueWords) * 4u;
    }

    // dynamic shared memory of k_dense: the planner info
    static size_t dense_smem(uint32_t blob_words) { return (size_t)((blob_words + 3u) & ~3u) * 4u; }

    // Enqueues the whole DP for n relations on `stream`.
    int enqueue(int n, DpMode mode, bool ccc, bool profile, uint32_t blob_words, std::string &err) {
        if (mode == kModeDpsize) return enqueue_dpsize(n, blob_words, err);
        const size_t smem = eval_smem(blob_words);
        const uint32_t max_block = reinterpret_cast<const DevHeader *>(h_blob)->max_block;
        const bool tree_mode = reinterpret_cast<const DevHeader *>(h_blob)->tree_mode != 0u;
        const int eval_max_blocks = sm_count * 4;
        const bool dense = dense_pairs(*reinterpret_cast<const DevHeader *>(h_blob));
        const int nw = ec_stride(reinterpret_cast<const DevHeader *>(h_blob)->n_ec) / 4;
        CK(cudaMemsetAsync(d_ctl, 0, kCtlClearBytes, stream));
        CK(cudaMemsetAsync(a.seen, 0, std::max<uint64_t>((1ull << n) / 8, 4), stream));
        // no winner and no share yet (k_dense leaves them so); sets of up to
        // kDenseWhole splits are one warp's, so smaller queries have no shares
        if (mode == kModeDpsub && dense && (1u << (n - 1)) > kDenseWhole) {
            CK(cudaMemsetAsync(a.ovf_off, 0, max_level_sets(n) * sizeof(uint32_t), stream));
            CK(cudaMemsetAsync(a.ovf_key, 0xFF, max_level_sets(n) * sizeof(unsigned long long), stream));
            CK(cudaMemsetAsync(a.ovf_first, 0xFF, max_level_sets(n) * sizeof(unsigned long long), stream));
        }
        n_kernels = 0;
        k_init_base<<<1, 32, 0, stream>>>(a.blob, a.memo, a.memo_left);
        n_kernels++;
        for (int k = 2; k <= n; k++) {
            uint64_t total = binom64(n, k);
            uint64_t threads_cap = (uint64_t)sm_count * 8 * kBlock;
            uint64_t threads = std::min<uint64_t>(threads_cap, (total + 3) / 4);
            threads = std::max<uint64_t>(threads, 32);
            uint32_t per_thread = (uint32_t)((total + threads - 1) / threads);
            uint32_t fblocks = (uint32_t)((total + (uint64_t)per_thread * kBlock - 1) / ((uint64_t)per_thread * kBlock));
            LevelCounters *lc = a.lvl + k;
            uint32_t *cur_sets = (k & 1) ? a.sets2 : a.sets;
            const uint32_t *prev_sets = (k & 1) ? a.sets : a.sets2;
            k_level_sets<<<fblocks, kBlock, 0, stream>>>(a.blob, a.binom, n, k, total, per_thread, prev_sets,
                                                         a.lvl + (k - 1), a.seen, cur_sets, lc);
            n_kernels += 2;
            int eblocks = (int)std::min<uint64_t>((uint64_t)eval_max_blocks, (total + kWarpsPerBlock - 1) / kWarpsPerBlock);
            CK(cudaEventRecordWithFlags(kev[2 * k], stream, cudaEventRecordExternal));
            if (mode == kModeDpsub && dense) {
                // whole sets per warp while a level has enough of them, shares
                // of a set otherwise: four for every warp, as long as the set's
                // table (150 instructions) is little against its splits (450 for
                // 32), and smaller ones only where warps would have none
                const uint32_t V = 1u << (k - 1);
                const uint64_t warps = (uint64_t)sm_count * 3 * kWarpsPerBlock;
                uint32_t share = 512u;
                while (share > 128u && total * V < share * warps) share /= 2u;
                while (share < 4096u && total * V >= 2u * share * 4u * warps) share *= 2u;
                const bool whole = V <= std::max(share, kDenseWhole);
                if (whole) share = V;
                (nw == 1 ? k_dense<1> : k_dense<2>)<<<sm_count * 3, kBlock, dense_smem(blob_words), stream>>>(
                    a.blob, blob_words, k, cur_sets, lc, a.memo, a.memo_left, a.ovf_key, a.ovf_first, a.ovf_off, a.glob, share);
            } else if (mode == kModeDpsub) {
                k_eval<kModeDpsub><<<eblocks, kBlock, smem, stream>>>(a.blob, blob_words, k, cur_sets, lc, a.memo,
                                                                      a.memo_left, a.ovf_set, a.ovf_P, a.ovf_off,
                                                                      a.ovf_key, a.ovf_first, a.glob, ccc);
            } else {
                // max useful group: pairs of a k-set are at least 2(k-1)
                int max_group = 1;
                while (max_group < 32 && max_group < 2 * (k - 1)) max_group <<= 1;
                const uint32_t target_lanes = (uint32_t)sm_count * 24u * 32u;
                int mblocks = (int)std::min<uint64_t>((uint64_t)sm_count * 4, (total * 32 + kBlock - 1) / kBlock);
                if (tree_mode) {
                    k_eval_tree<<<mblocks, kBlock, smem, stream>>>(a.blob, blob_words, k, cur_sets, lc, a.memo,
                                                                   a.memo_left, a.glob);
                } else {
                    k_eval_mpdp<<<mblocks, kBlock, smem, stream>>>(a.blob, blob_words, cur_sets, lc, a.memo,
                                                                   a.memo_left, a.ovf_set, a.ovf_P, a.ovf_off,
                                                                   a.ovf_key, a.ovf_first, a.glob, target_lanes,
                                                                   max_group);
                }
            }
            CK(cudaEventRecordWithFlags(kev[2 * k + 1], stream, cudaEventRecordExternal));
            bool may_overflow;
            if (mode == kModeDpsub) {
                may_overflow = !dense && ((1ull << k) - 2ull) > kOvfLimit;
            } else {
                // sum over blocks of 2^|b| - 2 with sum(|b| - 1) = k - 1 and
                // |b| <= the query graph's largest block
                int bmax = std::min<int>(std::max<int>((int)max_block, 2), k);
                uint64_t nblk = (uint64_t)(k - 1 + bmax - 2) / (uint64_t)(bmax - 1);
                may_overflow = nblk * ((1ull << bmax) - 2ull) > kOvfLimit;
            }
            if (may_overflow) {
                n_kernels += 2;
                int oblocks = sm_count * 4;
                if (mode == kModeDpsub) {
                    k_ovf_chunks<kModeDpsub><<<oblocks, kBlock, smem, stream>>>(
                        a.blob, blob_words, k, lc, a.memo, a.ovf_set, a.ovf_P, a.ovf_off, a.ovf_key, a.ovf_first,
                        a.glob, ccc);
                    k_ovf_finalize<kModeDpsub><<<sm_count, kBlock, smem, stream>>>(
                        a.blob, blob_words, lc, a.memo, a.memo_left, a.ovf_set, a.ovf_key, a.ovf_first);
                } else {
                    k_ovf_chunks<kModeMpdp><<<oblocks, kBlock, smem, stream>>>(
                        a.blob, blob_words, k, lc, a.memo, a.ovf_set, a.ovf_P, a.ovf_off, a.ovf_key, a.ovf_first,
                        a.glob, ccc);
                    k_ovf_finalize<kModeMpdp><<<sm_count, kBlock, smem, stream>>>(
                        a.blob, blob_words, lc, a.memo, a.memo_left, a.ovf_set, a.ovf_key, a.ovf_first);
                }
            }
        }
        uint32_t full = (n == 32) ? 0xFFFFFFFFu : ((1u << n) - 1u);
        k_extract<<<1, 32, 0, stream>>>(a.memo, a.memo_left, full, a.blob, a.tree, a.tree_n);
        n_kernels++;
        return 0;
    }

    int download(std::string &err) {
        CK(cudaMemcpyAsync(h_ctl, d_ctl, sizeof(EngineCtl), cudaMemcpyDeviceToHost, stream));
        return 0;
    }

    // Blocks of a tree query: enough lanes for every split of its widest level,
    // so that no level takes a second round, and no more, since a barrier
    // costs with its arrivals.  Up to kTreeClusterLevel blocks' worth run as
    // one cluster (a power of two of blocks), which the hardware synchronises:
    // star-12 (widest level 2772 splits, 11 blocks' worth) 66 us on 296 blocks,
    // 54 us in a cluster of 8.
    static int tree_grid(const TreePlan &plan, int n, int full) {
        uint64_t lanes = 1;
        for (int k = 2; k <= n; k++) lanes = std::max(lanes, (uint64_t)plan.count[k] * (uint64_t)(k - 1));
        const uint64_t blocks = (lanes + kBlock - 1) / kBlock;
        if (blocks > (uint64_t)kTreeClusterLevel) return (int)std::min<uint64_t>(blocks, (uint64_t)full);
        int grid = 1;
        while (grid < kTreeCluster && (uint64_t)grid < blocks) grid <<= 1;
        return std::min(grid, full);
    }

    // The whole tree-mode MPDP as one cooperative launch (k_dp_tree).  Returns
    // 0 and sets launched when the kernel was started.
    int launch_persistent(int n, uint32_t words, bool on_device, bool &launched, std::string &err) {
        launched = false;
        const size_t smem = (size_t)((words + 511u) & ~511u) * 4u;   // few sizes: the occupancy is looked up per size
        if (coop_off) return 0;
        const DevHeader *h = reinterpret_cast<const DevHeader *>(h_blob);
        TreePlan plan;
        const double sets = tree_level_counts(h, plan.count);
        int minb = force_minb;
        if (minb == 0) {
            const double per_level = sets / n;
            const Tuning &tu = g_tuning[device];
            minb = per_level <= tu.single_narrow_level_sets ? 2 : (per_level > tu.single_wide_level_sets ? 4 : 3);
        }
        const int layout = tree_layout(*h);
        static const void *const variants[3][3] = {
            {(const void *)k_dp_tree<2, 0>, (const void *)k_dp_tree<2, 1>, (const void *)k_dp_tree<2, 2>},
            {(const void *)k_dp_tree<3, 0>, (const void *)k_dp_tree<3, 1>, (const void *)k_dp_tree<3, 2>},
            // at 64 registers the class passes spill about 100 bytes and lose to
            // 3 blocks (star-20 with statistics 406 against 356 us)
            {(const void *)k_dp_tree<3, 0>, (const void *)k_dp_tree<3, 1>, (const void *)k_dp_tree<4, 2>}};
        const void *fn = variants[minb - 2][layout];
        const size_t key = smem * 16u + (size_t)minb * 3u + (size_t)layout;
        auto cb = coop_blocks.find(key);
        if (cb == coop_blocks.end()) {
            int blocks = 0, dev_coop = 0, occ = 0;
            cudaDeviceGetAttribute(&dev_coop, cudaDevAttrCooperativeLaunch, device);
            bool ok = dev_coop != 0;
            size_t &limit = smem_limit[fn];   // only ever raised: larger sizes stay launchable
            if (ok && smem > std::max<size_t>(limit, 48 * 1024)) {
                ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
                if (ok) limit = smem;
            }
            if (ok) ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kBlock, smem) == cudaSuccess;
            if (ok) blocks = occ * sm_count;
            cudaGetLastError();
            cb = coop_blocks.emplace(key, blocks).first;
        }
        const int full = cb->second;
        if (full <= 0) return 0;
        const bool bounded = gpuqo_b200_barrier_poll_limit > 0;   // the polled barrier on purpose
        const int grid = bounded || minb != 2 ? full : tree_grid(plan, n, full);
        const bool one_cluster = grid <= kTreeCluster && !bounded && minb == 2;
        if (!ctl_clean || bar_base > (1u << 30)) {
            CK(cudaMemsetAsync(d_ctl, 0, kCtlClearBytes, stream));   // counters, barrier words
            bar_base = 0u;
        }
        ctl_clean = false;   // until this launch is known to have finished
        if (!one_cluster && !on_device)
            CK(cudaMemcpyAsync(a.blob, h_blob, (size_t)words * 4u, cudaMemcpyHostToDevice, stream));
        CK(cudaEventRecord(ev0, stream));
        const uint32_t *blob_src = one_cluster && !on_device ? h_blob : a.blob;
        uint32_t bwords = words;
        plan_sets = sets;
        plan_pairs = 0;
        for (int k = 2; k <= n; k++) plan_pairs += (uint64_t)plan.count[k] * 2u * (uint64_t)(k - 1);
        bar_after = one_cluster ? bar_base : bar_base + (unsigned)n * (unsigned)grid;   // a barrier per level and the first
        *h_tree_n = 0;
        plan.near = near_order(1ull << n, sets, layout, l2_bytes) ? 1u : 0u;
        for (int k = 2; k <= n; k++)
            plan.group[k] = (uint8_t)tree_group(plan.count[k], k, (uint32_t)grid * kBlock, (uint32_t)std::min(grid, sm_count));
        unsigned poll_limit = (unsigned)std::max(0, gpuqo_b200_barrier_poll_limit);
        void *args[] = {&blob_src, &bwords, &a.memo, &a.memo_left, &a.sets, &a.sets2, &a.lvl,
                        &h_tree, &h_tree_n, &a.bar, &bar_base, &plan, &poll_limit};
        cudaError_t e;
        if (one_cluster) e = launch_cluster(fn, grid, smem, args, stream);
        else e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kBlock), args, smem, stream);
        if (e != cudaSuccess) {
            cudaGetLastError();
            coop_off = true;   // do not retry on this engine
            return 0;
        }
        n_kernels = 1;
        launched = true;
        return 0;
    }

    // waits for the last persistent run and reports whether its grid barrier
    // timed out (no plan arrived); a timeout latches the engine onto the
    // per-level launches (gpuqo_b200_reset_persistent clears it), so later calls
    // do not wait for another timeout first
    int barrier_failed(bool &failed, EngineStats &st, std::string &err) {
        CK(cudaStreamSynchronize(stream));
        CK(cudaGetLastError());
        failed = *const_cast<volatile int *>(h_tree_n) == 0;
        if (failed) {
            barrier_timed_out = true;
            st.barrier_timeouts++;
        } else {
            ctl_clean = true;
            bar_base = bar_after;
        }
        return 0;
    }

    // Stages the blob, makes sure the arena and the graph for (n, mode) exist.
    int prepare(const std::vector<uint32_t> &blob, int n, DpMode mode, bool ccc, bool profile, uint32_t &words,
                cudaGraphExec_t &exec, std::string &err) {
        if (int rc = init(err)) return rc;
        // the blob is staged in buckets of 512 words so that one captured
        // graph serves every query of the same size class
        words = ((uint32_t)blob.size() + 511u) & ~511u;
        if (int rc = ensure(n, words, err)) return rc;
        if (mode == kModeDpsize) {
            if (int rc = ensure_dpsize(n, err)) return rc;
            const std::vector<uint32_t> l1 = dpsize_level1_places(n);
            std::memcpy(h_level1, l1.data(), l1.size() * 4);
            CK(cudaMemcpyAsync(a.level1, h_level1, l1.size() * 4, cudaMemcpyHostToDevice, stream));
        }
        std::memset(h_blob, 0, words * 4);
        std::memcpy(h_blob, blob.data(), blob.size() * 4);
        const size_t smem = eval_smem(words);
        if (smem > 48 * 1024) {
            CK(cudaFuncSetAttribute(k_dpsize_eval, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CK(cudaFuncSetAttribute(k_eval<kModeDpsub>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CK(cudaFuncSetAttribute(k_eval<kModeMpdp>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CK(cudaFuncSetAttribute(k_eval_mpdp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CK(cudaFuncSetAttribute(k_eval_tree, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CK(cudaFuncSetAttribute(k_ovf_chunks<kModeDpsub>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CK(cudaFuncSetAttribute(k_ovf_chunks<kModeMpdp>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CK(cudaFuncSetAttribute(k_ovf_finalize<kModeDpsub>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CK(cudaFuncSetAttribute(k_ovf_finalize<kModeMpdp>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        }
        // the dense kernels are instantiated by the words of a class row
        const DevHeader *hb = reinterpret_cast<const DevHeader *>(h_blob);
        const int dense = (mode == kModeDpsub && dense_pairs(*hb)) ? ec_stride(hb->n_ec) / 4 : 0;
        if (dense) {
            // their pair tables beside the planner info: 47,360 bytes for 256
            // classes, the most there are
            const size_t table = kWarpsPerBlock * (dense == 1 ? sizeof(PairTable<1>) : sizeof(PairTable<2>));
            const void *fn = dense == 1 ? (const void *)k_dense<1> : (const void *)k_dense<2>;
            if (dense_smem(words) + table > 48 * 1024)
                CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dense_smem(words)));
        }
        CK(cudaMemcpyAsync(a.blob, h_blob, words * 4, cudaMemcpyHostToDevice, stream));
        exec = nullptr;
        const uint32_t mb = hb->max_block, tm = hb->tree_mode;
        GraphKey key{n, (((int)mode * 64 + (int)std::min<uint32_t>(mb, 63u)) * 2 + (int)(tm != 0u)) * 4 + dense,
                     ccc ? 1 : 0, (int)words};
        (void)profile;
        auto it = graphs.find(key);
        if (it != graphs.end()) {
            exec = it->second;
            n_kernels = graph_kernels[key];
            return 0;
        }
        CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        int rc = enqueue(n, mode, ccc, false, words, err);
        cudaGraph_t captured = nullptr;
        cudaError_t ce = cudaStreamEndCapture(stream, &captured);
        if (rc) {
            if (captured) cudaGraphDestroy(captured);
            return rc;
        }
        if (ce != cudaSuccess) {
            err = std::string("graph capture: ") + cudaGetErrorString(ce);
            return GPUQO_B200_ERR_CUDA;
        }
        CK(cudaGraphInstantiate(&exec, captured, 0));
        cudaGraphDestroy(captured);
        graphs[key] = exec;
        graph_kernels[key] = n_kernels;
        return 0;
    }

    int launch(cudaGraphExec_t exec, std::string &err) {
        ctl_clean = false;
        CK(cudaGraphLaunch(exec, stream));
        return 0;
    }

    // evaluate-kernel time of the last replay, from the per-level event
    // nodes captured in the graph
    int read_eval_events(int n, EngineStats &st, std::string &err) {
        for (int k = 2; k <= n; k++) {
            float kms = 0.f;
            CK(cudaEventElapsedTime(&kms, kev[2 * k], kev[2 * k + 1]));
            st.eval_kernel_ms += kms;
            st.eval_kernel_launches++;
        }
        return 0;
    }

    // Copies the plan and counters back and fills nodes / stats.
    int finish(int n, bool profile, std::vector<TreeNode> &nodes, EngineStats &st, std::string &err,
               bool persistent = false) {
        if (!persistent) {
            if (int rc = download(err)) return rc;
            CK(cudaStreamSynchronize(stream));
            CK(cudaGetLastError());
        }
        if (profile)
            if (int rc = read_eval_events(n, st, err)) return rc;
        int nn = *h_tree_n;
        if (nn != 2 * n - 1) {
            err = "plan extraction produced " + std::to_string(nn) + " nodes for " + std::to_string(n) + " relations";
            return GPUQO_B200_ERR_CUDA;
        }
        nodes.assign(h_tree, h_tree + nn);
        uint64_t csgs = 0, filt = 0;
        for (int k = 2; k <= n; k++) {
            if (!persistent) csgs += h_lvl[k].n_sets;
            filt += binom64(n, k);
            if (!persistent) st.fallback_sets += h_lvl[k].n_fb;
        }
        st.connected_sets += persistent ? (uint64_t)plan_sets - (uint64_t)n : csgs;
        st.filtered_subsets += filt;
        st.evaluated_pairs += persistent ? plan_pairs : h_glob->evaluated_pairs;
        st.memo_bytes = (1ull << n) * (sizeof(float4) + 4);
        st.kernel_launches += (uint32_t)n_kernels;
        return 0;
    }

    bool persistent_ok(const std::vector<uint32_t> &blob, DpMode mode) const {
        const DevHeader *h = reinterpret_cast<const DevHeader *>(blob.data());
        return gpuqo_b200_persistent != 0 && !coop_off && !barrier_timed_out && mode == kModeMpdp &&
               h->tree_mode != 0u;
    }

    // stage the blob without building a graph (persistent path); upload: on
    // the device too (launch_persistent copies it otherwise, where it has to)
    int stage(const std::vector<uint32_t> &blob, int n, bool upload, uint32_t &words, std::string &err) {
        if (int rc = init(err)) return rc;
        words = ((uint32_t)blob.size() + 3u) & ~3u;
        if (int rc = ensure(n, (words + 511u) & ~511u, err)) return rc;
        std::memcpy(h_blob, blob.data(), blob.size() * 4);
        for (uint32_t i = (uint32_t)blob.size(); i < words; i++) h_blob[i] = 0u;
        if (upload) CK(cudaMemcpyAsync(a.blob, h_blob, words * 4, cudaMemcpyHostToDevice, stream));
        return 0;
    }

    int run(const std::vector<uint32_t> &blob, int n, DpMode mode, bool ccc, bool profile,
            std::vector<TreeNode> &nodes, EngineStats &st, std::string &err) {
        if (persistent_ok(blob, mode)) {
            uint32_t pw;
            if (int rc = stage(blob, n, false, pw, err)) return rc;
            bool launched = false;
            if (int rc = launch_persistent(n, pw, false, launched, err)) return rc;
            CK(cudaEventRecord(ev1, stream));
            bool failed = true;
            if (launched) {
                if (int rc = barrier_failed(failed, st, err)) return rc;
            }
            if (launched && !failed) {
                if (int rc = finish(n, false, nodes, st, err, true)) return rc;
                float ms = 0.f;
                CK(cudaEventElapsedTime(&ms, ev0, ev1));
                st.device_ms += ms;
                st.eval_kernel_ms += ms;
                st.eval_kernel_launches += 1;
                return 0;
            }
            // not launched or the barrier timed out: per-level launches below
        }
        uint32_t words;
        cudaGraphExec_t exec;
        if (int rc = prepare(blob, n, mode, ccc, profile, words, exec, err)) return rc;
        CK(cudaEventRecord(ev0, stream));
        if (int rc = launch(exec, err)) return rc;
        CK(cudaEventRecord(ev1, stream));
        if (int rc = finish(n, profile, nodes, st, err)) return rc;
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, ev0, ev1));
        st.device_ms += ms;
        return 0;
    }

    // Device-resident timing: the planner info is uploaded once, then the DP
    // graph is replayed `iters` times with CUDA events around each replay on
    // the engine's stream; the L2 is flushed (a 256 MB write) between replays
    // outside the timed events.  Returns the mean device ms per replay.
    int time_resident(const std::vector<uint32_t> &blob, int n, DpMode mode, bool ccc, int warmup, int iters,
                      bool flush_l2, double &ms_per_iter, std::vector<TreeNode> &nodes, EngineStats &st,
                      std::string &err) {
        const size_t flush_floats = (256u << 20) / sizeof(float);
        if (persistent_ok(blob, mode)) {
            uint32_t pw;
            if (int rc = stage(blob, n, true, pw, err)) return rc;
            if (flush_l2 && !flush) CK(cudaMalloc(&flush, flush_floats * sizeof(float)));
            bool usable = true;   // every launch so far started and passed its barriers
            for (int i = 0; i < warmup && usable; i++) {
                bool launched = false, failed = false;
                if (int rc = launch_persistent(n, pw, true, launched, err)) return rc;
                if (launched)
                    if (int rc = barrier_failed(failed, st, err)) return rc;
                usable = launched && !failed;
            }
            double total = 0.0;
            for (int i = 0; usable && i < iters; i++) {
                if (flush_l2) CK(cudaMemsetAsync(flush, i & 0xFF, flush_floats * sizeof(float), stream));
                bool launched = false, failed = false;
                if (int rc = launch_persistent(n, pw, true, launched, err)) return rc;
                CK(cudaEventRecord(ev1, stream));
                CK(cudaEventSynchronize(ev1));
                float ms = 0.f;
                CK(cudaEventElapsedTime(&ms, ev0, ev1));
                total += ms;
                st.eval_kernel_ms += ms;
                st.eval_kernel_launches += 1;
                if (launched)
                    if (int rc = barrier_failed(failed, st, err)) return rc;
                usable = launched && !failed;
            }
            if (usable && iters > 0) {
                ms_per_iter = total / iters;
                st.device_ms += ms_per_iter;
                return finish(n, false, nodes, st, err, true);
            }
            st.eval_kernel_ms = 0.0;
            st.eval_kernel_launches = 0;
        }
        uint32_t words;
        cudaGraphExec_t exec;
        if (int rc = prepare(blob, n, mode, ccc, false, words, exec, err)) return rc;
        if (flush_l2 && !flush) CK(cudaMalloc(&flush, flush_floats * sizeof(float)));
        ctl_clean = false;
        for (int i = 0; i < warmup; i++) CK(cudaGraphLaunch(exec, stream));
        double total = 0.0;
        for (int i = 0; i < iters; i++) {
            if (flush_l2) CK(cudaMemsetAsync(flush, i & 0xFF, flush_floats * sizeof(float), stream));
            CK(cudaEventRecord(ev0, stream));
            CK(cudaGraphLaunch(exec, stream));
            CK(cudaEventRecord(ev1, stream));
            CK(cudaEventSynchronize(ev1));
            float ms = 0.f;
            CK(cudaEventElapsedTime(&ms, ev0, ev1));
            total += ms;
            if (int rc = read_eval_events(n, st, err)) return rc;
        }
        ms_per_iter = iters > 0 ? total / iters : 0.0;
        st.device_ms += ms_per_iter;
        return finish(n, false, nodes, st, err);
    }
};

// One engine of each kind per device, each device's engines and tuning
// record guarded by that device's mutex, so that host threads driving
// different devices (the batch and the server spread over several) do not
// wait for one another.
static std::mutex g_dev_mu[kMaxDevices];
static std::unique_ptr<Engine> g_engines[kMaxDevices];

// the calling thread's current device (a valid index of the engine tables)
static int current_device(int &dev, std::string &err) {
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        cudaGetLastError();
        err = std::string("cudaGetDevice: ") + cudaGetErrorString(e);
        return GPUQO_B200_ERR_CUDA;
    }
    if (dev < 0 || dev >= kMaxDevices) {
        err = "device index " + std::to_string(dev) + " beyond the library's " + std::to_string(kMaxDevices);
        return GPUQO_B200_ERR_CUDA;
    }
    return 0;
}

}  // namespace gqb

// ===========================================================================
// Entry point that allocates nothing.
//
// Some callers cannot allocate device memory: code that must not leak when
// Postgres aborts a query with elog(ERROR) (a longjmp past any cudaFree),
// processes whose device memory is owned by another pool, and paths with a
// fixed memory budget.  gpuqo_b200_run_noalloc serves them for queries of up
// to kNoAllocMaxRels relations: every scratch buffer of the DP (dense memo,
// level lists, overflow lists, counters, planner-info blob, plan nodes) is
// carved out of the one file-scope array below, which every GPU that loads
// this library holds until the process exits.  Host-side conversion uses
// fixed-size stack buffers; kernels are launched directly on the caller's
// stream (no graph, no events).
//
// In host code g_noalloc_scratch names a host-side stand-in, not the device
// array; its device address comes from cudaGetSymbolAddress, done once per
// device by the first call on that device (so make that first call before
// any stream capture).  All calls share the array: calls that overlap on the
// GPU race with each other.
// ===========================================================================
// Postgres cost GUCs (host_api.cpp / the backend), read the way setParams does
extern "C" double seq_page_cost, cpu_tuple_cost, cpu_operator_cost, disable_cost;
extern "C" int work_mem;
extern "C" bool enable_nestloop, enable_hashjoin;

namespace gqb {

constexpr int kNoAllocMaxRels = 18;
constexpr uint32_t kNoAllocMaxBlobWords = 6144;
constexpr uint64_t kNoAllocMaxSets = 48620;   // C(18, 9), the largest level

constexpr size_t na_align(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kNaMemo = 0;
constexpr size_t kNaMemoLeft = kNaMemo + na_align((1ull << kNoAllocMaxRels) * sizeof(float4));
constexpr size_t kNaSets = kNaMemoLeft + na_align((1ull << kNoAllocMaxRels) * sizeof(uint32_t));
constexpr size_t kNaOvfSet = kNaSets + na_align(kNoAllocMaxSets * 4);
constexpr size_t kNaOvfP = kNaOvfSet + na_align(kNoAllocMaxSets * 4);
constexpr size_t kNaOvfOff = kNaOvfP + na_align(kNoAllocMaxSets * 4);
constexpr size_t kNaOvfKey = kNaOvfOff + na_align(kNoAllocMaxSets * 4);
constexpr size_t kNaOvfFirst = kNaOvfKey + na_align(kNoAllocMaxSets * 8);
constexpr size_t kNaLvl = kNaOvfFirst + na_align(kNoAllocMaxSets * 8);
constexpr size_t kNaGlob = kNaLvl + na_align(33 * sizeof(LevelCounters));
constexpr size_t kNaBlob = kNaGlob + na_align(sizeof(GlobalCounters));
constexpr size_t kNaBinom = kNaBlob + na_align(kNoAllocMaxBlobWords * 4);
constexpr size_t kNaTree = kNaBinom + na_align(33 * 33 * 4);
constexpr size_t kNaTreeN = kNaTree + na_align(64 * sizeof(TreeNode));
constexpr size_t kNaTotal = kNaTreeN + na_align(sizeof(int));   // about 6.7 MB

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaTotal];

static std::mutex g_na_mu;
static unsigned char *g_na_ptr[64];   // device address of the scratch, per device
static bool g_na_ready[64];

// Once per device, with that device current: resolve the scratch address and
// fill the binomial table.  No allocation.
static int noalloc_setup(int dev) {
    std::lock_guard<std::mutex> lk(g_na_mu);
    if (g_na_ready[dev]) return 0;
    void *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || ptr == nullptr) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
        return GPUQO_B200_ERR_CUDA;
    }
    static uint32_t table[33 * 33];
    for (int i = 0; i <= 32; i++)
        for (int j = 0; j <= 32; j++) {
            uint64_t v = binom64(i, j);
            table[i * 33 + j] = v > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)v;
        }
    e = cudaMemcpy((unsigned char *)ptr + kNaBinom, table, sizeof(table), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: binomial table upload failed: %s\n", cudaGetErrorString(e));
        return GPUQO_B200_ERR_CUDA;
    }
    g_na_ptr[dev] = (unsigned char *)ptr;
    g_na_ready[dev] = true;
    return 0;
}

static inline uint64_t na_bms(const Bitmapset *b) { return (b && b->nwords > 0) ? b->words[0] : 0ull; }
static inline int na_popc(uint64_t x) { return __builtin_popcountll(x); }
static inline uint64_t na_pdep(uint64_t val, uint64_t mask) {
    uint64_t r = 0;
    for (uint64_t bb = 1; mask; bb += bb) {
        uint64_t low = mask & (~mask + 1);
        if (val & bb) r |= low;
        mask &= mask - 1;
    }
    return r;
}
static inline int na_ecidx(int l, int r, int size) {
    if (l > r) { int t = l; l = r; r = t; }
    return l * size - l * (l + 1) / 2 + (r - l - 1);
}

// GpuqoPlannerInfoC -> BFS-relabelled device blob in a caller buffer (the
// same relabelling as bfs_order/relabel/build_blob, in fixed-size storage).
// On failure prints the cause and returns its status code.
static int noalloc_blob(const GpuqoPlannerInfoC *c, uint32_t *blob, uint32_t &words, int *from_of_to) {
    const int n = c->n_rels;
    uint64_t edge[kNoAllocMaxRels];
    for (int i = 0; i < n; i++) {
        if (na_bms(c->base_rels[i].id) != (1ull << (i + 1))) {
            fprintf(stderr, "gpuqo_b200_run_noalloc: base relation %d does not carry relid bit %d\n", i, i + 1);
            return GPUQO_B200_ERR_ARGS;
        }
        edge[i] = na_bms(c->edge_table[i]);
    }
    // BFS order (gpuqo_bfs_indexing.cu:14-55)
    int queue[kNoAllocMaxRels * kNoAllocMaxRels + 1];
    int front = 0, back = 0, nt = 0;
    queue[back++] = 0;
    uint64_t seen = 2ull;
    while (front != back && nt < n) {
        int b = queue[front++];
        from_of_to[nt++] = b;
        uint64_t e = edge[b];
        while (e) {
            int next = __builtin_ffsll((long long)e) - 1;
            if (!(seen & (1ull << next)) && back < kNoAllocMaxRels * kNoAllocMaxRels) queue[back++] = next - 1;
            e &= ~(1ull << next);
        }
        seen |= edge[b];
    }
    if (nt != n) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: the query graph is disconnected\n");
        return GPUQO_B200_ERR_ARGS;
    }
    auto remap = [&](uint64_t m) {
        uint64_t o = 0;
        for (int t = 0; t < n; t++)
            if (m & (1ull << (from_of_to[t] + 1))) o |= 1ull << t;   // compact bit t
        return o;
    };
    int n_ec = 0, n_sels = 0, n_fks = 0;
    for (const EqClassInfo *ec = c->eq_classes; ec; ec = ec->next) {
        int s = na_popc(na_bms(ec->relids));
        n_ec++;
        n_sels += s * (s - 1) / 2;
        n_fks += s;
    }
    words = blob_words_for(n, n_ec, n_sels, n_fks);
    if (n_sels >= 65536 || n_fks >= 65536 || words > kNoAllocMaxBlobWords) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: the planner info needs %u words (%d equivalence classes, %d "
                        "selectivities, %d members); this entry point holds at most %u\n",
                words, n_ec, n_sels, n_fks, kNoAllocMaxBlobWords);
        return GPUQO_B200_ERR_TOO_LARGE;
    }
    for (uint32_t i = 0; i < words; i++) blob[i] = 0u;
    DevHeader *h = reinterpret_cast<DevHeader *>(blob);
    h->n = n;
    h->n_ec = n_ec;
    h->n_sels = n_sels;
    h->n_fks = n_fks;
    h->cpu_operator_cost = (float)cpu_operator_cost;
    h->cpu_tuple_cost = (float)cpu_tuple_cost;
    h->seq_page_cost = (float)seq_page_cost;
    h->disable_cost = (float)disable_cost;
    h->work_mem = work_mem;
    h->work_mem_bytes = work_mem_bytes_of(work_mem);
    h->enable_nestloop = enable_nestloop ? 1 : 0;
    h->enable_hashjoin = enable_hashjoin ? 1 : 0;
    h->composite_mask = 0;
    h->blob_words = words;
    long long width_sum = 0;
    bool width_ok = true;
    for (int t = 0; t < n; t++) {
        width_sum += c->base_rels[t].width;
        width_ok = width_ok && c->base_rels[t].width >= 0;
    }
    h->hz_packed = (width_ok && width_sum < (1ll << kWidthBits)) ? 1u : 0u;
    for (int t = 0; t < n; t++) {
        const BaseRelationC &b = c->base_rels[from_of_to[t]];
        h->adj[t] = (uint32_t)(remap(edge[from_of_to[t]]) & ~(1ull << t));
        h->rows[t] = b.rows;
        h->tuples[t] = b.tuples;
        h->startup[t] = b.cost.startup;
        h->total[t] = b.cost.total;
        h->width[t] = b.width;
        h->fksel[t] = (float)(1.0 / (double)fmaxf(1.0f, b.tuples));
    }
    DevInfoView v = make_view(blob);
    uint32_t *relids = const_cast<uint32_t *>(v.ec_relids);
    uint32_t *offs = const_cast<uint32_t *>(v.ec_off);
    float *sels = const_cast<float *>(v.sels);
    uint32_t *fks = const_cast<uint32_t *>(v.fks);
    DevVar *vars = const_cast<DevVar *>(v.vars);
    int i = 0, off_sels = 0, off_fks = 0;
    for (const EqClassInfo *ec = c->eq_classes; ec; ec = ec->next, i++) {
        uint64_t ecf = na_bms(ec->relids);     // Postgres bits
        uint64_t ect = remap(ecf);             // compact bits
        int s = na_popc(ecf);
        relids[i] = (uint32_t)ect;
        offs[i] = ((uint32_t)off_sels << 16) | (uint32_t)off_fks;
        for (int lt = 0; lt < s; lt++) {
            uint64_t id_lt = na_pdep(1ull << lt, ect);
            uint64_t id_lf = 1ull << (from_of_to[__builtin_ffsll((long long)id_lt) - 1] + 1);
            int lf = na_popc((id_lf - 1) & ecf);
            for (int rt = lt + 1; rt < s; rt++) {
                uint64_t id_rt = na_pdep(1ull << rt, ect);
                uint64_t id_rf = 1ull << (from_of_to[__builtin_ffsll((long long)id_rt) - 1] + 1);
                int rf = na_popc((id_rf - 1) & ecf);
                sels[off_sels + na_ecidx(lt, rt, s)] = ec->sels[na_ecidx(lf, rf, s)];
            }
            fks[off_fks + lt] = (uint32_t)remap(ec->fk ? na_bms(ec->fk[lf]) : 0ull);
            const VarInfo &vi = ec->vars[lf];
            DevVar &dv = vars[off_fks + lt];
            const int rel_t = __builtin_ffsll((long long)id_lt) - 1;   // compact index of this member
            dv.idx_rows = vi.index.rows;
            dv.idx_startup = vi.index.cost.startup;
            dv.idx_total = vi.index.cost.total;
            dv.flags = (vi.index.available ? 1u : 0u) | (vi.index.unique ? 2u : 0u);
            devvar_bucket_terms(dv, vi.stats.stadistinct, vi.stats.stanullfrac, vi.stats.mcvfreq, h->rows[rel_t],
                                h->tuples[rel_t]);
        }
        off_sels += s * (s - 1) / 2;
        off_fks += s;
    }
    fill_rel_ecs(v, n);
    fill_pair_sel(v);
    return 0;
}

}  // namespace gqb

extern "C" int gpuqo_b200_run_noalloc(int gpuqo_algorithm_arg, const GpuqoPlannerInfoC *info, void *cuda_stream,
                                      GpuqoB200PlanNode *out_nodes, int max_nodes, int *n_nodes) {
    using namespace gqb;
    if (!info || !out_nodes || !n_nodes) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: NULL argument\n");
        return GPUQO_B200_ERR_ARGS;
    }
    const int n = info->n_rels;
    if (n < 1 || n > kNoAllocMaxRels) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: %d relations; this entry point handles 1..%d\n", n,
                kNoAllocMaxRels);
        return GPUQO_B200_ERR_TOO_LARGE;
    }
    if (max_nodes < 2 * n - 1) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: output holds %d nodes, %d needed\n", max_nodes, 2 * n - 1);
        return GPUQO_B200_ERR_ARGS;
    }
    if (gpuqo_spanning_tree_enable) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: plans the query graph as given; gpuqo_spanning_tree_enable is "
                        "served by gpuqo_run\n");
        return GPUQO_B200_ERR_UNSUPPORTED;
    }
    DpMode mode;
    switch (gpuqo_algorithm_arg) {
    case GPUQO_CPU_DPSUB_BICC:
    case GPUQO_CPU_DPSUB_BICC_PARALLEL:
        mode = kModeMpdp;
        break;
    case GPUQO_CPU_DPSUB:
    case GPUQO_CPU_DPSUB_PARALLEL:
    case GPUQO_DPE_DPSUB:
        mode = kModeDpsub;
        break;
    case GPUQO_DPSUB:
        mode = gpuqo_dpsub_bicc_enable ? kModeMpdp : kModeDpsub;
        break;
    default:
        fprintf(stderr, "gpuqo_b200_run_noalloc: algorithm %d is not served by this entry point (DPsub and MPDP "
                        "only)\n", gpuqo_algorithm_arg);
        return GPUQO_B200_ERR_UNSUPPORTED;
    }
    uint32_t blob[kNoAllocMaxBlobWords];
    uint32_t words = 0;
    int from_of_to[kNoAllocMaxRels];
    if (int rc = noalloc_blob(info, blob, words, from_of_to)) return rc;
    // an error left pending by unrelated earlier work would otherwise be
    // reported as this call's own
    cudaGetLastError();
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GPUQO_B200_ERR_CUDA;
    if (int rc = noalloc_setup(dev)) return rc;
    unsigned char *base = g_na_ptr[dev];
    cudaStream_t stream = (cudaStream_t)cuda_stream;
    float4 *memo = (float4 *)(base + kNaMemo);
    uint32_t *memo_left = (uint32_t *)(base + kNaMemoLeft);
    uint32_t *sets = (uint32_t *)(base + kNaSets);
    uint32_t *ovf_set = (uint32_t *)(base + kNaOvfSet);
    uint32_t *ovf_P = (uint32_t *)(base + kNaOvfP);
    uint32_t *ovf_off = (uint32_t *)(base + kNaOvfOff);
    unsigned long long *ovf_key = (unsigned long long *)(base + kNaOvfKey);
    unsigned long long *ovf_first = (unsigned long long *)(base + kNaOvfFirst);
    LevelCounters *lvl = (LevelCounters *)(base + kNaLvl);
    GlobalCounters *glob = (GlobalCounters *)(base + kNaGlob);
    uint32_t *d_blob = (uint32_t *)(base + kNaBlob);
    uint32_t *binom = (uint32_t *)(base + kNaBinom);
    TreeNode *tree = (TreeNode *)(base + kNaTree);
    int *tree_n = (int *)(base + kNaTreeN);
    int sm_count = 148;
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    const int ccc = gpuqo_dpsub_ccc_enable ? 1 : 0;
    const size_t smem = (size_t)(((words + 3u) & ~3u) + kWarpsPerBlock * kQueueWords) * 4u;

    // every enqueue is checked where it is made, so a failure names its step
    auto failed = [&](cudaError_t e, const char *what) {
        if (e == cudaSuccess) return false;
        fprintf(stderr, "gpuqo_b200_run_noalloc: %s: %s\n", what, cudaGetErrorString(e));
        return true;
    };
    // counters start at zero on every call; the memo needs no clearing (only
    // entries written earlier in the same call are read)
    if (failed(cudaMemcpyAsync(d_blob, blob, words * 4, cudaMemcpyHostToDevice, stream), "planner info upload") ||
        failed(cudaMemsetAsync(lvl, 0, 33 * sizeof(LevelCounters), stream), "counter reset") ||
        failed(cudaMemsetAsync(glob, 0, sizeof(GlobalCounters), stream), "counter reset") ||
        failed(cudaMemsetAsync(tree_n, 0, sizeof(int), stream), "counter reset"))
        return GPUQO_B200_ERR_CUDA;
    k_init_base<<<1, 32, 0, stream>>>(d_blob, memo, memo_left);
    if (failed(cudaGetLastError(), "base relations launch")) return GPUQO_B200_ERR_CUDA;
    for (int k = 2; k <= n; k++) {
        uint64_t total = binom64(n, k);
        uint64_t threads = std::min<uint64_t>((uint64_t)sm_count * 8 * kBlock, (total + 3) / 4);
        threads = std::max<uint64_t>(threads, 32);
        uint32_t per_thread = (uint32_t)((total + threads - 1) / threads);
        uint32_t fblocks = (uint32_t)((total + (uint64_t)per_thread * kBlock - 1) / ((uint64_t)per_thread * kBlock));
        LevelCounters *lc = lvl + k;
        k_filter<<<fblocks, kBlock, 0, stream>>>(d_blob, binom, n, k, total, per_thread, sets, lc);
        int eblocks = (int)std::min<uint64_t>((uint64_t)sm_count * 4, (total + kWarpsPerBlock - 1) / kWarpsPerBlock);
        bool may_overflow = ((1ull << k) - 2ull) > kOvfLimit;
        if (mode == kModeDpsub) {
            k_eval<kModeDpsub><<<eblocks, kBlock, smem, stream>>>(d_blob, words, k, sets, lc, memo, memo_left, ovf_set,
                                                                  ovf_P, ovf_off, ovf_key, ovf_first, glob, ccc);
            if (may_overflow) {
                k_ovf_chunks<kModeDpsub><<<sm_count * 4, kBlock, smem, stream>>>(
                    d_blob, words, k, lc, memo, ovf_set, ovf_P, ovf_off, ovf_key, ovf_first, glob, ccc);
                k_ovf_finalize<kModeDpsub><<<sm_count, kBlock, smem, stream>>>(d_blob, words, lc, memo, memo_left,
                                                                               ovf_set, ovf_key, ovf_first);
            }
        } else {
            k_eval<kModeMpdp><<<eblocks, kBlock, smem, stream>>>(d_blob, words, k, sets, lc, memo, memo_left, ovf_set,
                                                                 ovf_P, ovf_off, ovf_key, ovf_first, glob, ccc);
            if (may_overflow) {
                k_ovf_chunks<kModeMpdp><<<sm_count * 4, kBlock, smem, stream>>>(
                    d_blob, words, k, lc, memo, ovf_set, ovf_P, ovf_off, ovf_key, ovf_first, glob, ccc);
                k_ovf_finalize<kModeMpdp><<<sm_count, kBlock, smem, stream>>>(d_blob, words, lc, memo, memo_left,
                                                                              ovf_set, ovf_key, ovf_first);
            }
        }
        if (failed(cudaGetLastError(), "level launch")) return GPUQO_B200_ERR_CUDA;
    }
    k_extract<<<1, 32, 0, stream>>>(memo, memo_left, (1u << n) - 1u, d_blob, tree, tree_n);
    if (failed(cudaGetLastError(), "plan extraction launch")) return GPUQO_B200_ERR_CUDA;
    TreeNode host_nodes[64];
    int host_n = 0;
    if (failed(cudaMemcpyAsync(host_nodes, tree, 64 * sizeof(TreeNode), cudaMemcpyDeviceToHost, stream),
               "plan download") ||
        failed(cudaMemcpyAsync(&host_n, tree_n, sizeof(int), cudaMemcpyDeviceToHost, stream), "plan download") ||
        failed(cudaStreamSynchronize(stream), "stream synchronisation"))
        return GPUQO_B200_ERR_CUDA;
    if (host_n != 2 * n - 1) {
        fprintf(stderr, "gpuqo_b200_run_noalloc: plan extraction produced %d nodes\n", host_n);
        return GPUQO_B200_ERR_CUDA;
    }
    for (int j = 0; j < host_n; j++) {
        uint64_t orig = 0;
        for (int t = 0; t < n; t++)
            if (host_nodes[j].set & (1u << t)) orig |= 1ull << (from_of_to[t] + 1);
        out_nodes[j].relids = orig;
        out_nodes[j].left = host_nodes[j].left;
        out_nodes[j].right = host_nodes[j].right;
        out_nodes[j].rows = host_nodes[j].rows;
        out_nodes[j].startup = host_nodes[j].startup;
        out_nodes[j].total = host_nodes[j].total;
        out_nodes[j].width = host_nodes[j].width;
    }
    *n_nodes = host_n;
    return GPUQO_B200_OK;
}

// ===========================================================================
// Batched MPDP: many independent queries level by level.  One wave packs the
// memos of its queries into one arena; per level one enumeration launch and
// one evaluation launch serve every query of the wave, so small queries no
// longer pay per-query launch latency.  Items of a level list are
// (query << 32 | set).  The planner info of each query stays in global
// memory (read through the read-only cache) because groups of one warp may
// belong to different queries.
// ===========================================================================
namespace gqb {

struct BatchQ {
    uint32_t blob_off;                 // word offset into the wave's blob buffer
    uint32_t n;
    uint32_t first_base;               // relations of the queries ahead: its first singleton in the level-1
                                       // list, and half the index of its first plan node
    uint32_t tree_tab;                 // word offset of its tree tables in the wave's blob buffer
    unsigned long long memo_off;       // entry offset into the memo arena
    unsigned long long seen_off;       // word offset into the dedup bitmap arena
};

// Sets of a level with more splits than their warp takes alone (kb_gen): all
// their splits are dealt out evenly over the grid after the level, in units
// of `unit` splits.  A set that finds the list full is evaluated by its warp.
struct BatchOvf {
    unsigned long long *item;          // [cap] query << 32 | set
    uint32_t *W;                       // [cap] unordered splits
    uint32_t *off;                     // [cap] first unit (increases with the index)
    unsigned long long *key;           // [cap] min (cost bits << 32 | candidate index) over the units
    uint32_t *nan_p;                   // [cap] lowest index of a NaN candidate
    uint32_t *done;                    // [cap] units finished
    uint32_t cap;
    uint32_t unit;
};

__global__ void kb_init(const BatchQ *__restrict__ qs, int nq, const uint32_t *__restrict__ blobs,
                        float4 *__restrict__ memo, uint32_t *__restrict__ memo_left,
                        unsigned long long *__restrict__ list1, LevelCounters *__restrict__ lvl1) {
    const int q = blockIdx.x;
    if (q >= nq) return;
    const BatchQ Q = qs[q];
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blobs + Q.blob_off);
    for (int i = threadIdx.x; i < (int)Q.n; i += blockDim.x) {
        memo[Q.memo_off + (1ull << i)] =
            base_entry(*h, i);
        memo_left[Q.memo_off + (1ull << i)] = 0u;
        list1[Q.first_base + i] = ((unsigned long long)q << 32) | (1u << i);
    }
    if (threadIdx.x == 0) atomicAdd(&lvl1->n_sets, Q.n);
}

// Warp-aggregated append of 64-bit items to a level list: lanes with ok set
// stage their item in the warp's 64-slot area; every 32 staged items take one
// atomicAdd on the level counter.  Call warp-uniformly; flush with
// stage_flush64 at the end.
__device__ __forceinline__ void stage_emit64(unsigned long long *st, uint32_t &cnt, bool ok,
                                             unsigned long long item, unsigned long long *out, LevelCounters *lc) {
    const int lane = threadIdx.x & 31;
    const uint32_t m = __ballot_sync(kFull, ok);
    if (ok) st[cnt + __popc(m & ((1u << lane) - 1u))] = item;
    cnt += __popc(m);
    __syncwarp();
    if (cnt >= 32) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&lc->n_sets, 32u);
        base = __shfl_sync(kFull, base, 0);
        out[base + lane] = st[lane];
        __syncwarp();
        if (lane < cnt - 32) st[lane] = st[32 + lane];
        cnt -= 32;
        __syncwarp();
    }
}

__device__ __forceinline__ void stage_flush64(unsigned long long *st, uint32_t &cnt, unsigned long long *out,
                                              LevelCounters *lc) {
    const int lane = threadIdx.x & 31;
    if (cnt > 0) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&lc->n_sets, cnt);
        base = __shfl_sync(kFull, base, 0);
        if (lane < cnt) out[base + lane] = st[lane];
    }
    cnt = 0;
    __syncwarp();
}

// connected k-sets of every query, by extension of its (k-1)-sets (c_prev
// items in prev); thread tid of nthreads (per-level launches)
__device__ __forceinline__ void batch_extend(const BatchQ *qs, const uint32_t *blobs, const unsigned long long *prev,
                                             uint32_t c_prev, uint32_t *seen, unsigned long long *out,
                                             LevelCounters *lc, unsigned long long *st, uint32_t tid,
                                             uint32_t nthreads) {
    uint32_t cnt = 0;
    const uint32_t rounds = (c_prev + nthreads - 1u) / nthreads;
    for (uint32_t r = 0; r < rounds; r++) {
        const uint32_t idx = tid + r * nthreads;
        uint32_t S = 0u, N = 0u, q = 0u;
        unsigned long long seen_off = 0;
        if (idx < c_prev) {
            const unsigned long long it = __ldcg(prev + idx);
            q = (uint32_t)(it >> 32);
            S = (uint32_t)it;
            const BatchQ Q = qs[q];
            const uint32_t *adj = reinterpret_cast<const DevHeader *>(blobs + Q.blob_off)->adj;
            seen_off = Q.seen_off;
            for (uint32_t x = S; x; x &= x - 1u) N |= __ldg(adj + lowest_idx(x));
            N &= ~S;
        }
        const int maxdeg = (int)__reduce_max_sync(kFull, (uint32_t)__popc(N));
        for (int j = 0; j < maxdeg; j++) {
            bool ok = N != 0u;
            unsigned long long item = 0;
            if (ok) {
                const uint32_t T = S | (N & (0u - N)), bm = 1u << (T & 31u);
                N &= N - 1u;
                ok = !(atomicOr(&seen[seen_off + (T >> 5)], bm) & bm);
                item = ((unsigned long long)q << 32) | T;
            }
            stage_emit64(st, cnt, ok, item, out, lc);
        }
    }
    stage_flush64(st, cnt, out, lc);
}

__global__ void __launch_bounds__(kBlock) kb_level_sets(const BatchQ *__restrict__ qs,
                                                        const uint32_t *__restrict__ blobs,
                                                        const unsigned long long *__restrict__ prev,
                                                        const LevelCounters *__restrict__ prev_lc,
                                                        uint32_t *__restrict__ seen,
                                                        unsigned long long *__restrict__ out,
                                                        LevelCounters *__restrict__ lc) {
    __shared__ unsigned long long stage[kWarpsPerBlock][64];
    const int warp = threadIdx.x >> 5;
    batch_extend(qs, blobs, prev, __ldcg(&prev_lc->n_sets), seen, out, lc, stage[warp],
                 blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// candidate c of a tree-shaped query: orientation c & 1 of the split at child
// end v
__device__ __forceinline__ void tree_cand(const DevHeader &h, uint32_t S, uint32_t v, uint32_t c, uint32_t &L,
                                          uint32_t &R, uint32_t &p, uint32_t &ecm, bool masked) {
    const TreeRows t = tree_rows(h, S);
    const uint2 e = *reinterpret_cast<const uint2 *>(t.row + 2u * v);
    const uint32_t comp = S & e.x, L0 = (e.y & kTreeLower) ? comp : S ^ comp;
    uint32_t p0, p1;
    tree_order(t, S, v, e.x, L0, h.index_order, p0, p1);
    L = (c & 1u) ? S ^ L0 : L0;
    R = S ^ L;
    p = (c & 1u) ? p1 : p0;
    ecm = masked ? reinterpret_cast<const TreeEdge *>(t.tab + tree_edge_off(t.n))[e.y & 31u].classes : 0u;
}

// the sets of one level of every query in groups of G lanes (per-level launches)
template <int G>
__device__ __forceinline__ void batch_groups(const BatchQ *qs, const uint32_t *blobs, uint32_t first, uint32_t stride,
                                             const unsigned long long *items, uint32_t count, int k, float4 *memo_all,
                                             uint32_t *memo_left_all, unsigned long long &pairs) {
    const int lane = threadIdx.x & 31;
    const int grp = lane / G, gl = lane % G;
    const uint32_t group_mask = (G == 32) ? kFull : (((1u << G) - 1u) << (grp * G));
    Blocks B;
    CycleCache cc;
    for (uint32_t base = first; base < count; base += stride) {
        const uint32_t i = base + (uint32_t)grp;
        const bool has = i < count;
        unsigned long long it = has ? __ldcg(items + i) : 0ull;
        const uint32_t q = (uint32_t)(it >> 32), S = (uint32_t)it;
        BatchQ Q;
        Q.blob_off = 0;
        Q.memo_off = 0;
        if (has) Q = qs[q];
        const DevInfoView d = make_view(blobs + Q.blob_off);
        const DevHeader &h = *d.h;
        float4 *memo = memo_all + Q.memo_off;
        uint32_t *memo_left = memo_left_all + Q.memo_off;
        const bool tree = has && h.tree_mode != 0u;
        const bool masked = tree && h.ec_masked != 0u;
        uint32_t P = 0;
        B.nb = 0;
        if (has) {
            if (tree) {
                P = 2u * (uint32_t)(k - 1);
            } else {
                find_blocks(S, h.adj, B);
                P = B.etotal;
            }
        }
        __syncwarp();
        const uint32_t iters = __reduce_max_sync(kFull, (P + G - 1u) / G);
        LaneBest best;
        best.init();
        uint32_t ends = S & (S - 1u), end_rank = 0u;   // child ends not passed yet, rank of the lowest
        int bcur = 0;
        for (uint32_t j = 0; j < iters; j++) {
            const uint32_t c = (uint32_t)gl + j * G;
            const bool active = has && c < P;
            uint32_t L = 0, R = 0, p = 0, ecm = 0;
            bool valid = false;
            if (active) {
                if (tree) {
                    for (; end_rank < (c >> 1); end_rank++) ends &= ends - 1u;
                    tree_cand(h, S, (uint32_t)lowest_idx(ends), c, L, R, p, ecm, masked);
                    valid = true;
                } else {
                    uint32_t key;
                    valid = mpdp_candidate(S, B, h.adj, c, bcur, L, R, key, cc);
                    p = valid ? key_index(h, key, L, S) : key;
                }
            }
            if (valid) {
                RelVal l = load_rel(memo, L, d.h->hz_packed), r = load_rel(memo, R, d.h->hz_packed);
                RelVal out = masked ? join_eval_t<true>(d, L, l, R, r, ecm) : join_eval_t<false>(d, L, l, R, r, 0u);
                best_update(best, p, L, out);
            }
        }
        uint32_t kh = (uint32_t)(best.key >> 32), kl = (uint32_t)best.key, fp = best.first_p;
#pragma unroll
        for (int off = G / 2; off >= 1; off >>= 1) {
            uint32_t oh = __shfl_xor_sync(kFull, kh, off);
            uint32_t ol = __shfl_xor_sync(kFull, kl, off);
            uint32_t of = __shfl_xor_sync(kFull, fp, off);
            if (oh < kh || (oh == kh && ol < kl)) {
                kh = oh;
                kl = ol;
            }
            if (of < fp) fp = of;
        }
        const bool nan_first = has && best.first_p == fp && best.first_nan();
        const unsigned nm = __ballot_sync(kFull, nan_first) & group_mask;
        const unsigned long long gkey = ((unsigned long long)kh << 32) | kl;
        if (has) {
            if (nm) {
                if (nan_first) memo_write(*d.h, memo, memo_left, S, best.nan_val, best.nan_left);
            } else if (best.key == gkey && best.key != ~0ull) {
                memo_write(*d.h, memo, memo_left, S, best.val, best.left);
            }
        }
        pairs += best.n_valid;
    }
}

__global__ void __launch_bounds__(kBlock) kb_eval(const BatchQ *__restrict__ qs, const uint32_t *__restrict__ blobs,
                                                  const unsigned long long *__restrict__ items,
                                                  const LevelCounters *__restrict__ lc, int k,
                                                  float4 *__restrict__ memo, uint32_t *__restrict__ memo_left,
                                                  GlobalCounters *__restrict__ glob, uint32_t target_lanes,
                                                  int max_group) {
    const uint32_t count = __ldcg(&lc->n_sets);
    if (count == 0u) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int G = 2;
    while (G < max_group && (uint64_t)count * (uint64_t)G < (uint64_t)target_lanes) G <<= 1;
    G = G <= 2 ? 2 : (G <= 8 ? 8 : 32);
    const uint32_t gwarp = blockIdx.x * kWarpsPerBlock + warp;
    const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
    unsigned long long pairs = 0;
    if (G == 2) batch_groups<2>(qs, blobs, gwarp * 16, nwarps * 16, items, count, k, memo, memo_left, pairs);
    else if (G == 8) batch_groups<8>(qs, blobs, gwarp * 4, nwarps * 4, items, count, k, memo, memo_left, pairs);
    else batch_groups<32>(qs, blobs, gwarp, nwarps, items, count, k, memo, memo_left, pairs);
    pairs = __reduce_add_sync(kFull, (uint32_t)pairs);
    if (lane == 0 && pairs) atomicAdd(&glob->evaluated_pairs, pairs);
}

// kb_gen: a wave of queries whose graphs have cycles, or one such query (ONE:
// its planner info in shared memory), in ONE cooperative, persistent launch.
// Per level k: one warp per connected k-set evaluates it (dp_general.cuh)
// while the far end of the grid enumerates level k + 1, also one warp per set
// and one lane per neighbour, deduplicated in a bitmap of all subsets, or for
// a cactus graph, whose connected sets are counted beforehand and whose sides
// need no test, in a table of 2^table_log2 words when that is smaller (a
// 30-relation bitmap takes 30 us to clear).  Sets with more splits than `limit` go to the
// overflow list; after the barrier their splits are dealt out evenly, and the
// warp that finishes a set's last unit writes its entry.
// Bound: latency on the graphs planned exactly at this size (few sets per
// level): list entry, block search (about 2 us for 30 relations), two memo
// entries, cost, barrier.  Before, every lane searched the blocks in local
// memory, one warp walked up to 2048 candidates of a set, and both orientations
// were costed apart.  Device time: key cycle-30 1031 -> 402 us, random graphs
// of 16 relations with statistics (0.59 and 0.72 M pairs) 3304 / 3360 -> 510 /
// 552 us.
__device__ __forceinline__ uint32_t gen_units(const BatchOvf &ovf, uint32_t W) { return (W + ovf.unit - 1u) / ovf.unit; }

// connected (k+1)-sets from the c_prev k-sets in prev; `warp` of nwarps
__device__ __forceinline__ void gen_extend(const BatchQ *qs, const uint32_t *blobs, const uint32_t *own_adj,
                                           const unsigned long long *prev, uint32_t c_prev, uint32_t *seen,
                                           uint32_t table_log2, unsigned long long *out, LevelCounters *lc,
                                           unsigned long long *st, uint32_t warp, uint32_t nwarps) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t cnt = 0;
    for (uint32_t i = warp; i < c_prev; i += nwarps) {
        const unsigned long long it = __ldcg(prev + i);
        const uint32_t q = (uint32_t)(it >> 32), S = (uint32_t)it;
        const uint32_t *adj = own_adj;
        unsigned long long seen_off = 0;
        uint32_t n;
        if (own_adj) {
            n = reinterpret_cast<const DevHeader *>(blobs)->n;
        } else {
            const BatchQ Q = qs[q];
            adj = reinterpret_cast<const DevHeader *>(blobs + Q.blob_off)->adj;
            seen_off = Q.seen_off;
            n = Q.n;
        }
        const uint32_t bit = 1u << lane, T = S | bit;
        bool ok = lane < n && !(S & bit) && (adj[lane] & S) != 0u;
        if (ok && table_log2) {
            // at most half full: an empty or the set's own slot is found
            uint32_t at = (T * 0x9E3779B1u) >> (32u - table_log2);
            for (uint32_t probe = 0; probe < (1u << table_log2); probe++, at = (at + 1u) & ((1u << table_log2) - 1u)) {
                const uint32_t old = atomicCAS(seen + at, 0u, T);
                ok = old == 0u;
                if (ok || old == T) break;
            }
        } else if (ok) {
            const uint32_t bm = 1u << (T & 31u);
            ok = !(atomicOr(&seen[seen_off + (T >> 5)], bm) & bm);
        }
        stage_emit64(st, cnt, ok, ((unsigned long long)q << 32) | T, out, lc);
    }
    stage_flush64(st, cnt, out, lc);
}

template <bool ONE>
__device__ __forceinline__ void gen_overflow(const BatchQ *qs, const uint32_t *blobs, const uint32_t *own,
                                             LevelCounters *lc, float4 *memo_all, uint32_t *memo_left_all,
                                             const uint32_t *seen_all, const BatchOvf &ovf, GenScratch &ws,
                                             uint32_t gwarp, uint32_t nwarps, uint32_t &pairs) {
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned long long packed = __ldcg(&lc->ovf_packed);
    uint32_t n = (uint32_t)(packed >> 40), total = (uint32_t)(packed & 0xFFFFFFFFFFull);
    if (n > ovf.cap) {
        n = ovf.cap;
        total = __ldcg(ovf.off + n - 1u) + gen_units(ovf, __ldcg(ovf.W + n - 1u));
    }
    const uint32_t per = (total + nwarps - 1u) / nwarps;
    uint32_t first = gwarp * per;
    const uint32_t last = min(first + per, total);
    if (first >= last) return;
    uint32_t lo_i = 0u, hi_i = n - 1u;   // largest idx with off[idx] <= first
    while (lo_i < hi_i) {
        const uint32_t mid = (lo_i + hi_i + 1u) >> 1;
        if (__ldcg(ovf.off + mid) <= first) lo_i = mid;
        else hi_i = mid - 1u;
    }
    for (uint32_t idx = lo_i; first < last; idx++) {
        const unsigned long long it = __ldcg(ovf.item + idx);
        const uint32_t q = (uint32_t)(it >> 32), S = (uint32_t)it;
        const uint32_t W = __ldcg(ovf.W + idx), o = __ldcg(ovf.off + idx), units = gen_units(ovf, W);
        BatchQ Q = {};
        if (!ONE) Q = qs[q];
        const DevInfoView d = make_view(ONE ? own : blobs + Q.blob_off);
        float4 *memo = memo_all + Q.memo_off;
        const uint32_t *seen = seen_all + Q.seen_off;
        gen_blocks(S, d.h->adj, ws);
        GenBest best;
        best.init();
        int width = 0;
        const uint32_t end = min(units, last - o);
        gen_range(d, ws, S, (first - o) * ovf.unit, min(W, end * ovf.unit), memo, seen, best, width);
        pairs += best.pairs;
        uint32_t ord, p;
        gen_winner(*d.h, ws, S, best, true, ord, p);
        const uint32_t nan_p = __reduce_min_sync(kFull, best.nan_p);
        uint32_t finished = 0u;
        if (lane == 0u) {
            if (ord != kFull) atomicMin(ovf.key + idx, ((unsigned long long)ord << 32) | p);
            if (nan_p != kFull) atomicMin(ovf.nan_p + idx, nan_p);
            __threadfence();
            const uint32_t mine = end - (first - o);
            finished = atomicAdd(ovf.done + idx, mine) + mine == units ? 1u : 0u;
            __threadfence();
        }
        finished = __shfl_sync(kFull, finished, 0);
        __syncwarp();
        if (finished) {
            const uint32_t gnan = __ldcg(ovf.nan_p + idx);
            uint32_t w = (uint32_t)__ldcg(ovf.key + idx);
            if (gnan != kFull && gnan == gen_first(S, d.h->index_order, seen)) w = gnan;
            gen_write_index(d, ws, S, w, memo, memo_left_all + Q.memo_off);
        }
        first = o + units;
    }
}

template <bool ONE>
__global__ void __launch_bounds__(kBlock, 2) kb_gen(const BatchQ *__restrict__ qs, int nq, int maxn,
                                                    const uint32_t *__restrict__ blobs, uint32_t blob_words,
                                                    float4 *__restrict__ memo, uint32_t *__restrict__ memo_left,
                                                    uint32_t *seen, unsigned long long *__restrict__ listA,
                                                    unsigned long long *__restrict__ listB,
                                                    LevelCounters *__restrict__ lvl, GlobalCounters *__restrict__ glob,
                                                    TreeNode *__restrict__ tree, int *__restrict__ tree_n,
                                                    unsigned *__restrict__ bar, BatchOvf ovf, uint32_t table_log2,
                                                    unsigned poll_limit) {
    extern __shared__ __align__(16) unsigned char gsm[];
    __shared__ unsigned long long stage[kWarpsPerBlock][64];
    const unsigned max_polls = barrier_polls(poll_limit);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GenScratch &ws = reinterpret_cast<GenScratch *>(gsm)[warp];
    uint32_t *own = nullptr;
    if (ONE) {
        own = reinterpret_cast<uint32_t *>(gsm + kWarpsPerBlock * sizeof(GenScratch));
        load_blob_to_smem(blobs, blob_words, own);
    }
    unsigned long long *st = stage[warp];
    const uint32_t gwarp = blockIdx.x * kWarpsPerBlock + warp;
    const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
    unsigned long long pairs = 0;
    unsigned epoch = 0;   // grid barriers passed (thread 0)
    // small queries run as one cluster, synchronised in hardware
    const bool cluster = ONE && cluster_blocks() == gridDim.x;
    auto barrier = [&]() -> bool {
        if (ONE && cluster) {
            cluster_barrier();
            return true;
        }
        return grid_barrier<ONE>(bar, epoch, max_polls);
    };

    // phase 0: base relations (gpuqo_cpu_sequential.cu:80-92) and level-2 sets
    // (each edge once, from its lower end), entered into the bitmap
    {
        uint32_t cnt = 0;
        for (uint32_t q = gwarp; q < (uint32_t)nq; q += nwarps) {
            const BatchQ Q = qs[q];
            const DevHeader *h = reinterpret_cast<const DevHeader *>(ONE ? own : blobs + Q.blob_off);
            uint32_t nb = 0u;
            if (lane < (int)Q.n) {
                memo[Q.memo_off + (1ull << lane)] = base_entry(*h, lane);
                memo_left[Q.memo_off + (1ull << lane)] = 0u;
                if (!table_log2) atomicOr(seen + Q.seen_off + ((1u << lane) >> 5), 1u << ((1u << lane) & 31u));
                nb = h->adj[lane] & ~((2u << lane) - 1u);
            }
            const int maxdeg = (int)__reduce_max_sync(kFull, (uint32_t)__popc(nb));
            for (int j = 0; j < maxdeg; j++) {
                const bool ok = nb != 0u;
                const uint32_t T = (1u << lane) | (nb & (0u - nb));
                nb &= nb - 1u;
                if (ok && !table_log2) atomicOr(seen + Q.seen_off + (T >> 5), 1u << (T & 31u));
                stage_emit64(st, cnt, ok, ((unsigned long long)q << 32) | T, listA, lvl + 2);
            }
        }
        stage_flush64(st, cnt, listA, lvl + 2);
    }
    if (!barrier()) return;

    for (int k = 2; k <= maxn; k++) {
        unsigned long long *cur = (k & 1) ? listB : listA;
        unsigned long long *nxt = (k & 1) ? listA : listB;
        LevelCounters *lk = lvl + k;
        const uint32_t count = __ldcg(&lk->n_sets);
        // enumeration from the far end of the grid, evaluation from the start
        if (k < maxn)
            gen_extend(qs, ONE ? own : blobs, ONE ? reinterpret_cast<const DevHeader *>(own)->adj : nullptr, cur, count,
                       seen, table_log2, nxt, lk + 1, st, nwarps - 1u - gwarp, nwarps);
        // Splits a warp takes alone: 4 rounds of its lanes per set it holds.
        // The overflow phase costs about two barriers and another block search
        // per share.
        const uint32_t limit = min(2048u, 128u * ((count + nwarps - 1u) / nwarps));
        uint32_t found = 0u;
        for (uint32_t i = gwarp; i < count; i += nwarps) {
            const unsigned long long it = __ldcg(cur + i);
            const uint32_t q = (uint32_t)(it >> 32), S = (uint32_t)it;
            BatchQ Q = {};
            if (!ONE) Q = qs[q];
            const DevInfoView d = make_view(ONE ? own : blobs + Q.blob_off);
            if (d.h->tree_tab != 0u) {
                gen_cactus_set(d, cactus_view(reinterpret_cast<const uint32_t *>(d.h) + d.h->tree_tab, d.h->n_ec),
                               plain_params(*d.h), ws, S, memo + Q.memo_off, memo_left + Q.memo_off, found);
                continue;
            }
            gen_blocks(S, d.h->adj, ws);
            const uint32_t W = ws.half[ws.nb];
            if (W > limit && ovf.cap != 0u) {
                // one packed atomic assigns the list index and the first unit
                // in the same order
                uint32_t idx = 0u;
                if (lane == 0) {
                    const unsigned long long old = atomicAdd(&lk->ovf_packed, (1ull << 40) | gen_units(ovf, W));
                    idx = (uint32_t)(old >> 40);
                    if (idx < ovf.cap) {
                        ovf.item[idx] = it;
                        ovf.W[idx] = W;
                        ovf.off[idx] = (uint32_t)(old & 0xFFFFFFFFFFull);
                        ovf.key[idx] = ~0ull;
                        ovf.nan_p[idx] = kFull;
                        ovf.done[idx] = 0u;
                    }
                }
                if (__shfl_sync(kFull, idx, 0) < ovf.cap) continue;
            }
            gen_set(d, ws, S, memo + Q.memo_off, memo_left + Q.memo_off, seen + Q.seen_off, found);
        }
        if (!barrier()) return;
        // the counter is final after the barrier: every block takes the same branch
        if (ovf.cap != 0u && (uint32_t)(__ldcg(&lk->ovf_packed) >> 40) != 0u) {
            gen_overflow<ONE>(qs, blobs, own, lk, memo, memo_left, seen, ovf, ws, gwarp, nwarps, found);
            if (!barrier()) return;
        }
        pairs += found;
    }

    for (uint32_t q = gwarp; q < (uint32_t)nq; q += nwarps) {
        const BatchQ Q = qs[q];
        const uint32_t full = (Q.n == 32) ? 0xFFFFFFFFu : ((1u << Q.n) - 1u);
        const uint32_t wmask =
            reinterpret_cast<const DevHeader *>(ONE ? own : blobs + Q.blob_off)->hz_packed ? kWidthMask : 0xFFFFFFFFu;
        extract_plan(memo + Q.memo_off, memo_left + Q.memo_off, full, wmask, ws.queue, tree + 2u * Q.first_base, tree_n + q);
    }
    for (int off = 16; off >= 1; off >>= 1) pairs += __shfl_xor_sync(kFull, pairs, off);
    if (lane == 0 && pairs) atomicAdd(&glob->evaluated_pairs, pairs);
}

__global__ void kb_extract(const BatchQ *__restrict__ qs, int nq, const uint32_t *__restrict__ blobs,
                           const float4 *__restrict__ memo, const uint32_t *__restrict__ memo_left,
                           TreeNode *__restrict__ out, int *__restrict__ n_out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nq) return;
    const BatchQ Q = qs[q];
    const uint32_t wmask =
        reinterpret_cast<const DevHeader *>(blobs + Q.blob_off)->hz_packed ? kWidthMask : 0xFFFFFFFFu;
    const uint32_t full = (Q.n == 32) ? 0xFFFFFFFFu : ((1u << Q.n) - 1u);
    TreeNode *o = out + 2u * Q.first_base;
    const float4 *m = memo + Q.memo_off;
    const uint32_t *ml = memo_left + Q.memo_off;
    int n = 0;
    uint32_t stack_set[64];
    int stack_parent[64], stack_side[64];
    int sp = 0;
    stack_set[sp] = full;
    stack_parent[sp] = -1;
    stack_side[sp] = 0;
    sp++;
    while (sp > 0 && n < 64) {
        sp--;
        uint32_t s = stack_set[sp];
        int parent = stack_parent[sp], side = stack_side[sp];
        float4 v = __ldcg(m + s);
        TreeNode t;
        t.set = s;
        t.left = -1;
        t.right = -1;
        t.rows = v.x;
        t.startup = v.y;
        t.total = v.z;
        t.width = (int)(__float_as_uint(v.w) & wmask);
        int me = n++;
        o[me] = t;
        if (parent >= 0) {
            if (side == 0) o[parent].left = me;
            else o[parent].right = me;
        }
        uint32_t l = __ldcg(ml + s) & s;
        if (__popc(s) > 1 && l != 0u && l != s && sp + 2 <= 64) {
            stack_set[sp] = s ^ l;
            stack_parent[sp] = me;
            stack_side[sp] = 1;
            sp++;
            stack_set[sp] = l;
            stack_parent[sp] = me;
            stack_side[sp] = 0;
            sp++;
        }
    }
    n_out[q] = n;
}

// kb_dp: a wave of tree-shaped queries in ONE cooperative, persistent launch.
// Phase 0 writes every query's base relations and emits its level-2 sets
// (one warp per query, one lane per relation: each edge once, from its lower
// end).  Then, per level k, the grid evaluates level k of every query
// (tree_set, the planner infos in global memory) while it enumerates level
// k+1, with a grid barrier between levels; the plans are extracted (one warp
// per query) after the last level.  The grid barrier is bounded
// (grid_barrier); on timeout the host reruns the wave with per-level launches.
// Bound: issue in the wide levels, the chain item -> query -> tables -> memo
// entries in the narrow ones.  With both orientations of a split taken
// together and no class pass (see k_dp_tree), device time of 96 queries of 10 to
// 20 relations (77 M pairs, its wave of cycles included) 2230 -> 1000 us, of
// 512 queries of 8 to 16 (23.7 M pairs) 1040 -> 600 us.
__device__ __forceinline__ void batch_tree_enum(const BatchQ *qs, const uint32_t *blobs, const unsigned long long *prev,
                                                uint32_t c_prev, bool near, unsigned long long *out,
                                                LevelCounters *lc, uint32_t tid, uint32_t nthreads) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t first = tid & ~31u; first < c_prev; first += nthreads) {
        const uint32_t idx = first + (tid & 31u);
        const unsigned long long it = idx < c_prev ? __ldcg(prev + idx) : 0ull;
        const uint32_t *adj = reinterpret_cast<const DevHeader *>(blobs + qs[it >> 32].blob_off)->adj;
        uint32_t ext = tree_extensions((uint32_t)it, near, [&](int v) { return __ldg(adj + v); });
        const uint32_t cnt = (uint32_t)__popc(ext);
        uint32_t incl = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(kFull, incl, off);
            if (lane >= (uint32_t)off) incl += o;
        }
        uint32_t base = 0u;
        if (lane == 31u && incl) base = atomicAdd(&lc->n_sets, incl);
        uint32_t at = __shfl_sync(kFull, base, 31) + incl - cnt;
        for (; ext; ext &= ext - 1u) out[at++] = it | (ext & (0u - ext));
    }
}

template <int LAYOUT>
__device__ __forceinline__ void batch_tree_level(const BatchQ *qs, const uint32_t *blobs, uint32_t gwarp, uint32_t nwarps,
                                                 const unsigned long long *items, uint32_t count, int k, int G,
                                                 float4 *memo, uint32_t *memo_left) {
    const uint32_t per_warp = 32u / (uint32_t)G, grp = (threadIdx.x & 31u) / (uint32_t)G;
    for (uint32_t base = gwarp * per_warp; base < count; base += nwarps * per_warp) {
        const bool has = base + grp < count;
        const unsigned long long it = has ? __ldcg(items + base + grp) : 0ull;
        const uint32_t S = (uint32_t)it;
        const BatchQ Q = qs[it >> 32];
        const DevInfoView d = make_view(blobs + Q.blob_off);
        TreeRows t;
        t.tab = blobs + Q.tree_tab;
        t.n = (int)Q.n;
        t.row = t.tab + (has ? t.tab[lowest_idx(S)] : 0u);
        tree_set<LAYOUT>(d, plain_params(*d.h), t, S, has, k, G, memo + Q.memo_off, memo_left + Q.memo_off);
    }
}

template <int LAYOUT>
__global__ void __launch_bounds__(kBlock, 3) kb_dp(const BatchQ *__restrict__ qs, int nq, int maxn,
                                                   const uint32_t *__restrict__ blobs, float4 *__restrict__ memo,
                                                   uint32_t *__restrict__ memo_left,
                                                   unsigned long long *__restrict__ listA,
                                                   unsigned long long *__restrict__ listB,
                                                   LevelCounters *__restrict__ lvl, GlobalCounters *__restrict__ glob,
                                                   TreeNode *__restrict__ tree, int *__restrict__ tree_n,
                                                   unsigned *__restrict__ bar, uint32_t sms, uint32_t near,
                                                   unsigned poll_limit) {
    const unsigned max_polls = barrier_polls(poll_limit);
    __shared__ unsigned long long stage[kWarpsPerBlock][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long *st = stage[warp];
    const uint32_t gwarp = blockIdx.x * kWarpsPerBlock + warp;
    const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nthreads = gridDim.x * blockDim.x;
    unsigned long long pairs = 0;
    unsigned epoch = 0;   // grid barriers passed (thread 0)

    // phase 0 (gpuqo_cpu_sequential.cu:80-92 for the base entries)
    {
        uint32_t cnt = 0;
        for (uint32_t q = gwarp; q < (uint32_t)nq; q += nwarps) {
            const BatchQ Q = qs[q];
            const DevHeader *h = reinterpret_cast<const DevHeader *>(blobs + Q.blob_off);
            const int v = lane;
            uint32_t nb = 0u;
            if (v < (int)Q.n) {
                memo[Q.memo_off + (1ull << v)] = base_entry(*h, v);
                memo_left[Q.memo_off + (1ull << v)] = 0u;
                nb = __ldg(h->adj + v) & ~((2u << v) - 1u);
            }
            const int deg = __popc(nb);
            const int maxdeg = (int)__reduce_max_sync(kFull, (uint32_t)deg);
            for (int j = 0; j < maxdeg; j++) {
                const bool ok = j < deg;
                unsigned long long item = 0;
                if (ok) {
                    const int u = __ffs(nb) - 1;
                    nb &= nb - 1u;
                    item = ((unsigned long long)q << 32) | (1u << v) | (1u << u);
                }
                stage_emit64(st, cnt, ok, item, listA, lvl + 2);
            }
        }
        stage_flush64(st, cnt, listA, lvl + 2);
    }
    if (!grid_barrier<false>(bar, epoch, max_polls)) return;

    for (int k = 2; k <= maxn; k++) {
        unsigned long long *cur = (k & 1) ? listB : listA;
        unsigned long long *nxt = (k & 1) ? listA : listB;
        const uint32_t count = __ldcg(&lvl[k].n_sets);
        // enumeration from the far end of the grid, evaluation from the start
        if (k < maxn) batch_tree_enum(qs, blobs, cur, count, near != 0u, nxt, lvl + k + 1, nthreads - 1u - tid, nthreads);
        batch_tree_level<LAYOUT>(qs, blobs, gwarp, nwarps, cur, count, k, tree_group(count, k, nthreads, sms), memo,
                                 memo_left);
        pairs += (unsigned long long)count * 2ull * (unsigned long long)(k - 1);   // every split edge, both orientations
        if (!grid_barrier<false>(bar, epoch, max_polls)) return;
    }

    for (uint32_t q = gwarp; q < (uint32_t)nq; q += nwarps) {
        const BatchQ Q = qs[q];
        const uint32_t full = (Q.n == 32) ? 0xFFFFFFFFu : ((1u << Q.n) - 1u);
        const uint32_t wmask =
            reinterpret_cast<const DevHeader *>(blobs + Q.blob_off)->hz_packed ? kWidthMask : 0xFFFFFFFFu;
        extract_plan(memo + Q.memo_off, memo_left + Q.memo_off, full, wmask, reinterpret_cast<uint32_t *>(st),
                     tree + 2u * Q.first_base, tree_n + q);
    }
    if (tid == 0) glob->evaluated_pairs = pairs;
}

// Candidate bound of a query for the batch (the batch has no overflow path):
// sum over blocks of 2^|b| - 2 with |b| <= the graph's largest block.
static uint64_t mpdp_candidate_bound(int n, int max_block) {
    int bmax = std::min(std::max(max_block, 2), std::max(n, 2));
    uint64_t nblk = (uint64_t)(n - 1 + bmax - 2) / (uint64_t)(bmax - 1);
    return nblk * ((1ull << bmax) - 2ull);
}

bool batch_eligible(const std::vector<uint32_t> &blob) {
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob.data());
    return h->n >= 1 && h->n <= 30;
}

// true when some set of the query may have more candidates than one group
// evaluates: those sets need the overflow phase of kb_gen
static bool batch_needs_ovf(const std::vector<uint32_t> &blob) {
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob.data());
    return mpdp_candidate_bound(h->n, (int)h->max_block) > kOvfLimit;
}

constexpr uint64_t kBatchOvfCap = 1ull << 22;   // overflow list entries per wave (32 B each)

// Connected sets of a tree-shaped query graph (its connected subtrees): with
// f(v) = prod over children c of (1 + f(c)) for the tree rooted at relation
// 0, the count is the sum of f(v).  Exact, O(n).
static double tree_connected_sets(const DevHeader *h) {
    const int n = h->n;
    int order[32], parent[32], m = 0;
    uint32_t seen = 1u;
    order[m++] = 0;
    parent[0] = -1;
    for (int i = 0; i < m; i++) {
        uint32_t nb = h->adj[order[i]] & ~seen;
        seen |= nb;
        while (nb) {
            const int c = __builtin_ctz(nb);
            nb &= nb - 1u;
            parent[c] = order[i];
            order[m++] = c;
        }
    }
    double f[32], total = 0.0;
    for (int i = 0; i < n; i++) f[i] = 1.0;
    for (int i = m - 1; i >= 0; i--) {
        const int v = order[i];
        total += f[v];
        if (parent[v] >= 0) f[parent[v]] *= 1.0 + f[v];
    }
    return total;
}

// A tree-shaped query with this many connected sets fills the GPU on its own:
// the single-query kernel (k_dp_tree, planner info in shared memory) then
// evaluates more pairs per second than a batch wave, so the batch hands it over.
// (Tuning::batch_single_sets, 2^20 until the autotuner measures it)
static bool batch_prefers_single(const std::vector<uint32_t> &blob, int device) {
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob.data());
    return h->tree_mode != 0u && gpuqo_b200_persistent != 0 &&
           tree_connected_sets(h) > g_tuning[device].batch_single_sets;
}

double engine_work_estimate(const std::vector<uint32_t> &blob) {
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob.data());
    const double n = (double)h->n;
    if (h->tree_mode) return tree_connected_sets(h) * 2.0 * std::max(n - 1.0, 1.0);
    return std::ldexp(1.0, h->n) * n;
}

uint64_t batch_query_bytes(int n) {
    const uint64_t slots = 1ull << n;
    return slots * (sizeof(float4) + 4) + slots / 8 + 2 * max_level_sets(n) * 8 + 64 * sizeof(TreeNode) + 4096;
}

// control words of a wave: cleared with one memset, brought back with its plans
struct alignas(16) BatchCtl {
    LevelCounters lvl[33];
    GlobalCounters glob;
    unsigned bar[4];                   // grid barrier: arrivals, -, error flag
};

// dynamic shared memory of kb_gen besides the planner info
constexpr size_t kGenSmem = kWarpsPerBlock * sizeof(GenScratch);
// beside it kb_gen has the list staging (8 bytes x 64 per warp) and the
// barrier's verdict as static shared memory: without opt-in 48 KB in all
static_assert(kGenSmem + kWarpsPerBlock * 64 * 8 + 16 <= 48 * 1024 && sizeof(GenScratch) % 16 == 0, "kb_gen shared memory");

struct BatchEngine {
    int device = -1, sm_count = 148, l2_bytes = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // arena (grown on demand), each buffer with its own capacity: one that
    // could not be allocated has none, whatever the others hold
    uint64_t cap_memo = 0, cap_left = 0, cap_seen = 0, cap_listA = 0, cap_listB = 0;
    float4 *memo = nullptr;
    uint32_t *memo_left = nullptr, *blobs = nullptr, *seen = nullptr;
    unsigned long long *listA = nullptr, *listB = nullptr;
    BatchQ *qs = nullptr;
    TreeNode *tree = nullptr;
    int *tree_n = nullptr;
    LevelCounters *lvl = nullptr;                // views into d_out
    GlobalCounters *glob = nullptr;
    unsigned *bar = nullptr;
    // device side of a wave's two copies: descriptors and planner infos in
    // (qs, blobs), control words, node counts and plans out (BatchCtl, tree_n, tree)
    unsigned char *d_in = nullptr, *d_out = nullptr;
    uint64_t cap_in = 0, cap_out = 0;
    int coop_grid = -1;                          // co-resident blocks of kb_gen<false> (0: no cooperative launch)
    int coop_grid_tree[3] = {-1, -1, -1};        // co-resident blocks of kb_dp by layout (tree_layout)
    std::map<size_t, int> coop_one;              // dynamic shared bytes -> co-resident blocks of kb_gen<true>
    bool barrier_timed_out = false;              // a grid barrier gave up: per-level launches until reset
    BatchOvf ovf{};                              // overflow list of kb_gen
    uint64_t cap_ovf[6] = {};                    // of its arrays
    void *flush = nullptr;                       // L2 flush buffer (device-resident timing only)
    // pinned staging of a wave: planner infos and descriptors in, plans and
    // counters out (grown on demand; the copies are truly asynchronous)
    unsigned char *h_in = nullptr, *h_out = nullptr;
    size_t cap_h_in = 0, cap_h_out = 0;
    bool ready = false;                          // init has come to its end

    static int grow_pinned(unsigned char *&p, size_t &cap, size_t bytes, std::string &err) {
        if (bytes <= cap) return 0;
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
        CK(cudaMallocHost(&p, bytes));
        cap = bytes;
        return 0;
    }

    int init(std::string &err) {
        if (ready) return 0;
        CK(cudaGetDevice(&device));
        CK(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
        CK(cudaDeviceGetAttribute(&l2_bytes, cudaDevAttrL2CacheSize, device));
        if (!stream) CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        if (!ev0) CK(cudaEventCreate(&ev0));
        if (!ev1) CK(cudaEventCreate(&ev1));
        int dev_coop = 0, occ = 0, occ_tree[3] = {0, 0, 0};
        cudaDeviceGetAttribute(&dev_coop, cudaDevAttrCooperativeLaunch, device);
        no_cooperative();
        if (dev_coop &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kb_gen<false>, kBlock, kGenSmem) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_tree[0], kb_dp<0>, kBlock, 0) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_tree[1], kb_dp<1>, kBlock, 0) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_tree[2], kb_dp<2>, kBlock, 0) == cudaSuccess) {
            coop_grid = occ * sm_count;
            for (int i = 0; i < 3; i++) coop_grid_tree[i] = occ_tree[i] * sm_count;
        }
        cudaGetLastError();
        ready = true;
        return 0;
    }

    void no_cooperative() { coop_grid = coop_grid_tree[0] = coop_grid_tree[1] = coop_grid_tree[2] = 0; }

    // per-level launches of one wave (the queries, blobs and arena are staged)
    uint32_t enqueue_levels(int nq, int maxn, uint64_t seen_words) {
        cudaMemsetAsync(d_out, 0, sizeof(BatchCtl), stream);
        cudaMemsetAsync(seen, 0, seen_words * 4, stream);
        kb_init<<<nq, 32, 0, stream>>>(qs, nq, blobs, memo, memo_left, listA, lvl + 1);
        uint32_t kernels = 1;
        const uint32_t target_lanes = (uint32_t)sm_count * 24u * 32u;
        for (int k = 2; k <= maxn; k++) {
            unsigned long long *prev = (k & 1) ? listB : listA;
            unsigned long long *cur = (k & 1) ? listA : listB;
            kb_level_sets<<<sm_count * 8, kBlock, 0, stream>>>(qs, blobs, prev, lvl + (k - 1), seen, cur, lvl + k);
            int max_group = 1;
            while (max_group < 32 && max_group < 2 * (k - 1)) max_group <<= 1;
            kb_eval<<<sm_count * 4, kBlock, 0, stream>>>(qs, blobs, cur, lvl + k, k, memo, memo_left, glob,
                                                         target_lanes, max_group);
            kernels += 2;
        }
        kb_extract<<<(nq + 127) / 128, 128, 0, stream>>>(qs, nq, blobs, memo, memo_left, tree, tree_n);
        return kernels + 1;
    }

    // co-resident blocks of kb_gen<true> with a planner info of `words` words,
    // 0 when two of them do not fit an SM (about 75 KB of planner info, an
    // 18-relation clique has 13 KB) or cooperative launches are not possible
    int one_grid(uint32_t words) {
        const size_t smem = kGenSmem + (size_t)words * 4u;
        if (coop_grid <= 0 || smem > 100u * 1024u) return 0;
        auto it = coop_one.find(smem);
        if (it == coop_one.end()) {
            int occ = 0;
            if (cudaFuncSetAttribute(kb_gen<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024) != cudaSuccess ||
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kb_gen<true>, kBlock, smem) != cudaSuccess)
                occ = 0;
            cudaGetLastError();
            it = coop_one.emplace(smem, occ * sm_count).first;
        }
        return it->second;
    }

    // the wave as one cooperative launch: kb_dp<layout> when every query is
    // tree-shaped (layout: the least of the queries' tree_layout), else kb_gen
    // (layout < 0; kb_gen<true> for one query); false when it could not start
    bool enqueue_persistent(int nq, int maxn, uint32_t words, uint64_t slots, uint64_t seen_words, int layout,
                            uint32_t cactus_sets) {
        const bool tree_only = layout >= 0;
        const int one = (!tree_only && nq == 1) ? one_grid(words) : 0;
        int grid = tree_only ? coop_grid_tree[layout] : (one > 0 ? one : coop_grid);
        // one cactus query: a table of twice its connected sets, and a cluster
        // when the widest levels (taken as twice the average) leave its warps
        // idle, half for the sets and half for their extensions
        uint32_t table_log2 = 0;
        bool cluster = false;
        if (one > 0 && cactus_sets != 0u && cactus_sets < (1u << 30)) {
            uint32_t l = 6;
            while ((1ull << l) < 2ull * cactus_sets) l++;
            if ((1ull << l) <= seen_words / 4) table_log2 = l;
            const double warps = 4.0 * (double)cactus_sets / (double)maxn;
            cluster = gpuqo_b200_barrier_poll_limit <= 0 && warps <= 2.0 * kTreeCluster * kWarpsPerBlock;
            if (cluster) grid = std::min(grid, kTreeCluster);
        }
        if (grid <= 0 || gpuqo_b200_persistent == 0 || barrier_timed_out) return false;
        cudaMemsetAsync(d_out, 0, sizeof(BatchCtl), stream);
        if (!tree_only) cudaMemsetAsync(seen, 0, table_log2 ? (size_t)4 << table_log2 : seen_words * 4, stream);
        unsigned poll_limit = (unsigned)std::max(0, gpuqo_b200_barrier_poll_limit);
        cudaError_t e;
        if (tree_only) {
            static const void *const variants[3] = {(const void *)kb_dp<0>, (const void *)kb_dp<1>, (const void *)kb_dp<2>};
            uint32_t sms = (uint32_t)sm_count, near = near_order(slots, 0.0, layout, l2_bytes) ? 1u : 0u;
            void *args[] = {&qs, &nq, &maxn, &blobs, &memo, &memo_left, &listA, &listB,
                            &lvl, &glob, &tree, &tree_n, &bar, &sms, &near, &poll_limit};
            e = cudaLaunchCooperativeKernel(variants[layout], dim3(grid), dim3(kBlock), args, 0, stream);
        } else {
            void *args[] = {&qs, &nq, &maxn, &blobs, &words, &memo, &memo_left, &seen, &listA, &listB,
                            &lvl, &glob, &tree, &tree_n, &bar, &ovf, &table_log2, &poll_limit};
            const void *fn = one > 0 ? (const void *)kb_gen<true> : (const void *)kb_gen<false>;
            const size_t smem = kGenSmem + (one > 0 ? (size_t)words * 4u : 0u);
            e = cluster ? launch_cluster(fn, grid, smem, args, stream)
                        : cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kBlock), args, smem, stream);
        }
        if (e != cudaSuccess) {
            cudaGetLastError();
            no_cooperative();
            return false;
        }
        return true;
    }

    // grows geometrically (twice the old capacity when that is more than the
    // need) so that waves of changing composition do not reallocate the arena
    // every time; falls back to the exact need when the larger block does
    // not fit
    template <class T> int grow(T *&p, uint64_t &cap, uint64_t need, std::string &err) {
        if (need <= cap) return 0;
        const uint64_t want = std::max(need, 2 * cap);
        cap = 0;
        release(p);
        if (want > need && cudaMalloc(&p, want * sizeof(T)) == cudaSuccess) {
            cap = want;
            return 0;
        }
        cudaGetLastError();
        p = nullptr;
        CK(cudaMalloc(&p, need * sizeof(T)));
        cap = need;
        return 0;
    }

    bool persistent_ready() const {
        return coop_grid > 0 && coop_grid_tree[0] > 0 && gpuqo_b200_persistent != 0 && !barrier_timed_out;
    }

    // One wave: all queries' memos fit.  wb: per query planner-info blob.
    // Queries that this wave cannot finish (sets beyond the group limit, whose
    // splits the per-level launches do not deal out) are listed in redo
    // (wave-local indices) for the single-query engine.
    int run_wave(const std::vector<const std::vector<uint32_t> *> &wb, std::vector<std::vector<TreeNode>> &out,
                 std::vector<int> &redo, EngineStats &st, double &ms, std::string &err) {
        redo.clear();
        std::vector<int> need_ovf;
        for (int q = 0; q < (int)wb.size(); q++)
            if (batch_needs_ovf(*wb[q])) need_ovf.push_back(q);
        if (!need_ovf.empty() && !persistent_ready()) {
            // per-level launches cannot split a set: those queries run alone
            std::vector<const std::vector<uint32_t> *> rest;
            std::vector<int> idx;
            size_t j = 0;
            for (int q = 0; q < (int)wb.size(); q++) {
                if (j < need_ovf.size() && need_ovf[j] == q) {
                    j++;
                    continue;
                }
                rest.push_back(wb[q]);
                idx.push_back(q);
            }
            out.assign(wb.size(), {});
            redo = need_ovf;
            ms = 0.0;
            if (rest.empty()) return 0;
            std::vector<std::vector<TreeNode>> rout;
            if (int rc = stage_and_run(rest, rout, st, ms, err)) return rc;
            for (size_t i = 0; i < idx.size(); i++) out[idx[i]] = std::move(rout[i]);
            return 0;
        }
        return stage_and_run(wb, out, st, ms, err);
    }

    int stage_and_run(const std::vector<const std::vector<uint32_t> *> &wb, std::vector<std::vector<TreeNode>> &out,
                      EngineStats &st, double &ms, std::string &err) {
        const int nq = (int)wb.size();
        std::vector<BatchQ> hq(nq);
        uint64_t slots = 0, words = 0, seen_words = 0, items = 0, base = 0, ovf_need = 0;
        int maxn = 0;
        int layout = kTreePlain;   // of a wave of trees; -1: a graph with cycles among the queries
        uint32_t cactus_sets = 0;  // connected sets of the last query if it is a cactus graph with cycles
        for (int q = 0; q < nq; q++) {
            const DevHeader *h = reinterpret_cast<const DevHeader *>(wb[q]->data());
            const int n = h->n;
            hq[q].blob_off = (uint32_t)words;
            hq[q].n = (uint32_t)n;
            hq[q].first_base = (uint32_t)base;
            hq[q].tree_tab = hq[q].blob_off + h->tree_tab;
            hq[q].memo_off = slots;
            hq[q].seen_off = seen_words;
            words += (wb[q]->size() + 3) & ~(size_t)3;
            slots += 1ull << n;
            seen_words += std::max<uint64_t>((1ull << n) / 32, 1);
            items += max_level_sets(n);
            base += (uint64_t)n;
            maxn = std::max(maxn, n);
            if (batch_needs_ovf(*wb[q])) ovf_need += max_level_sets(n);
            layout = h->tree_mode != 0u ? std::min(layout, tree_layout(*h)) : -1;
            if (h->tree_mode == 0u && h->tree_tab != 0u)
                cactus_sets = reinterpret_cast<const CactusHead *>(wb[q]->data() + h->tree_tab)->n_sets;
        }
        items = std::max(items, base);
        ovf_need = std::min(ovf_need, kBatchOvfCap);
        if (int rc = over_budget(slots * (sizeof(float4) + 4) + words * 4 + seen_words * 4 + items * 16 + ovf_need * 32,
                                 "the batch wave's arena", err))
            return rc;
        if (int rc = grow(memo, cap_memo, slots, err)) return rc;
        if (int rc = grow(memo_left, cap_left, slots, err)) return rc;
        if (int rc = grow(seen, cap_seen, seen_words, err)) return rc;
        if (int rc = grow(listA, cap_listA, items, err)) return rc;
        if (int rc = grow(listB, cap_listB, items, err)) return rc;
        if (int rc = grow(ovf.item, cap_ovf[0], ovf_need, err)) return rc;
        if (int rc = grow(ovf.W, cap_ovf[1], ovf_need, err)) return rc;
        if (int rc = grow(ovf.off, cap_ovf[2], ovf_need, err)) return rc;
        if (int rc = grow(ovf.key, cap_ovf[3], ovf_need, err)) return rc;
        if (int rc = grow(ovf.nan_p, cap_ovf[4], ovf_need, err)) return rc;
        if (int rc = grow(ovf.done, cap_ovf[5], ovf_need, err)) return rc;
        ovf.cap = (uint32_t)ovf_need;
        // units of the overflow shares: small enough to spread a level evenly,
        // large enough that a level's units number below 2^32 (at most 2^22
        // listed sets of 2^(n - 1) splits)
        ovf.unit = maxn <= 24 ? 32u : (maxn <= 26 ? 1024u : 8192u);
        const size_t in_q = (size_t)nq * sizeof(BatchQ), in_bytes = in_q + (size_t)words * 4;
        const size_t o_n = sizeof(BatchCtl), o_tree = (o_n + (size_t)nq * sizeof(int) + 15) & ~(size_t)15,
                     o_end = o_tree + 2 * (size_t)base * sizeof(TreeNode);
        if (int rc = grow(d_in, cap_in, in_bytes, err)) return rc;
        if (int rc = grow(d_out, cap_out, o_end, err)) return rc;
        qs = reinterpret_cast<BatchQ *>(d_in);
        blobs = reinterpret_cast<uint32_t *>(d_in + in_q);
        lvl = reinterpret_cast<BatchCtl *>(d_out)->lvl;
        glob = &reinterpret_cast<BatchCtl *>(d_out)->glob;
        bar = reinterpret_cast<BatchCtl *>(d_out)->bar;
        tree_n = reinterpret_cast<int *>(d_out + o_n);
        tree = reinterpret_cast<TreeNode *>(d_out + o_tree);
        // stage the descriptors and the planner infos in pinned memory (the
        // previous wave's copies ended with its synchronisation)
        if (int rc = grow_pinned(h_in, cap_h_in, in_bytes, err)) return rc;
        if (int rc = grow_pinned(h_out, cap_h_out, o_end, err)) return rc;
        std::memcpy(h_in, hq.data(), in_q);
        uint32_t *hblob = reinterpret_cast<uint32_t *>(h_in + in_q);
        for (int q = 0; q < nq; q++) {
            const size_t len = wb[q]->size(), padded = (len + 3) & ~(size_t)3;
            std::memcpy(hblob + hq[q].blob_off, wb[q]->data(), len * 4);
            std::memset(hblob + hq[q].blob_off + len, 0, (padded - len) * 4);
        }
        CK(cudaMemcpyAsync(d_in, h_in, in_bytes, cudaMemcpyHostToDevice, stream));
        // control words and plans come back in one copy
        const BatchCtl &ctl = *reinterpret_cast<const BatchCtl *>(h_out);
        auto download = [&]() -> int {
            CK(cudaMemcpyAsync(h_out, d_out, o_end, cudaMemcpyDeviceToHost, stream));
            CK(cudaStreamSynchronize(stream));
            CK(cudaGetLastError());
            return 0;
        };
        uint32_t kernels = 1;
        CK(cudaEventRecord(ev0, stream));
        bool persistent = enqueue_persistent(nq, maxn, (uint32_t)words, slots, seen_words, layout, cactus_sets);
        CK(cudaGetLastError());
        if (!persistent) kernels = enqueue_levels(nq, maxn, seen_words);
        CK(cudaGetLastError());
        CK(cudaEventRecord(ev1, stream));
        if (int rc = download()) return rc;
        if (persistent && ctl.bar[2] != 0u) {   // barrier timed out: rerun with per-level launches
            persistent = false;
            barrier_timed_out = true;           // and use them until gpuqo_b200_reset_persistent
            st.barrier_timeouts++;
            CK(cudaEventRecord(ev0, stream));
            kernels = enqueue_levels(nq, maxn, seen_words);
            CK(cudaGetLastError());
            CK(cudaEventRecord(ev1, stream));
            if (int rc = download()) return rc;
        }
        const TreeNode *htree = reinterpret_cast<const TreeNode *>(h_out + o_tree);
        const int *hn = reinterpret_cast<const int *>(h_out + o_n);
        float fms = 0.f;
        CK(cudaEventElapsedTime(&fms, ev0, ev1));
        ms = fms;
        out.resize(nq);
        for (int q = 0; q < nq; q++) {
            if (hn[q] != 2 * (int)hq[q].n - 1) {
                err = "batched plan extraction produced " + std::to_string(hn[q]) + " nodes";
                return GPUQO_B200_ERR_CUDA;
            }
            out[q].assign(htree + 2 * (size_t)hq[q].first_base, htree + 2 * (size_t)hq[q].first_base + hn[q]);
        }
        for (int k = 2; k <= maxn; k++) st.connected_sets += ctl.lvl[k].n_sets;
        st.evaluated_pairs += ctl.glob.evaluated_pairs;
        st.memo_bytes = std::max<uint64_t>(st.memo_bytes, slots * (sizeof(float4) + 4));
        st.device_ms += fms;
        st.kernel_launches += kernels;
        return 0;
    }
};

static std::unique_ptr<BatchEngine> g_batch[kMaxDevices];

int engine_run_batch(const std::vector<const std::vector<uint32_t> *> &blobs, uint64_t wave_bytes,
                     std::vector<std::vector<TreeNode>> &out, EngineStats &st, std::vector<double> &wave_ms,
                     std::string &err) {
    int dev = 0;
    if (int rc = current_device(dev, err)) return rc;
    std::lock_guard<std::mutex> lk(g_dev_mu[dev]);
    auto &be = g_batch[dev];
    if (!be) be.reset(new BatchEngine());
    if (int rc = be->init(err)) return rc;
    out.assign(blobs.size(), {});
    auto &eng = g_engines[dev];
    // large tree-shaped queries: one persistent single-query launch each
    std::vector<size_t> rest;
    for (size_t i = 0; i < blobs.size(); i++) {
        if (!batch_prefers_single(*blobs[i], dev)) {
            rest.push_back(i);
            continue;
        }
        if (!eng) eng.reset(new Engine());
        const int n = reinterpret_cast<const DevHeader *>(blobs[i]->data())->n;
        const double before = st.device_ms;
        if (int rc = eng->run(*blobs[i], n, kModeMpdp, true, false, out[i], st, err)) return rc;
        st.handoff_ms += st.device_ms - before;
    }
    // tree-shaped queries first (waves of kb_dp), then the others (kb_gen); the
    // order within each part is the caller's (largest first)
    std::stable_partition(rest.begin(), rest.end(), [&](size_t i) {
        return reinterpret_cast<const DevHeader *>(blobs[i]->data())->tree_mode != 0u;
    });
    // waves: consecutive queries while the wave's memory stays within budget
    // and its queries are all tree-shaped or all not
    size_t r = 0;
    while (r < rest.size()) {
        std::vector<const std::vector<uint32_t> *> wave;
        std::vector<size_t> idx;
        uint64_t bytes = 0;
        const bool wave_tree = reinterpret_cast<const DevHeader *>(blobs[rest[r]]->data())->tree_mode != 0u;
        while (r < rest.size()) {
            const size_t i = rest[r];
            const DevHeader *hi = reinterpret_cast<const DevHeader *>(blobs[i]->data());
            const int n = hi->n;
            const uint64_t b = batch_query_bytes(n);
            if (!wave.empty() && (bytes + b > wave_bytes || (hi->tree_mode != 0u) != wave_tree)) break;
            wave.push_back(blobs[i]);
            idx.push_back(i);
            bytes += b;
            r++;
        }
        std::vector<std::vector<TreeNode>> wout;
        std::vector<int> redo;
        double ms = 0;
        if (int rc = be->run_wave(wave, wout, redo, st, ms, err)) return rc;
        wave_ms.push_back(ms);
        for (size_t j = 0; j < idx.size(); j++) out[idx[j]] = std::move(wout[j]);
        if (!redo.empty()) {
            if (!eng) eng.reset(new Engine());
            for (int r : redo) {
                const std::vector<uint32_t> &b = *wave[r];
                const int n = reinterpret_cast<const DevHeader *>(b.data())->n;
                std::vector<TreeNode> nodes;
                if (int rc = eng->run(b, n, kModeMpdp, true, false, nodes, st, err)) return rc;
                out[idx[r]] = std::move(nodes);
            }
        }
    }
    return 0;
}


// One exact DP.  Tree-shaped graphs run k_dp_tree (Engine); other graphs
// under MPDP enumeration (MPDP, and plain DPsub on valid pairs) run as a
// one-query wave of the general persistent kernel kb_gen<true>, which has the
// overflow phases in the same launch; the per-level launches of Engine serve
// the rest (plain all-subsets DPsub, no cooperative launch,
// gpuqo_b200_persistent = 0).
int engine_run(const std::vector<uint32_t> &blob, int n, DpMode mode, bool ccc, bool profile,
               std::vector<TreeNode> &nodes, EngineStats &stats, std::string &err) {
    if (n < 1 || n > 31) {
        err = "exact DP supports 1..31 relations";
        return GPUQO_B200_ERR_TOO_LARGE;
    }
    int dev = 0;
    if (int rc = current_device(dev, err)) return rc;
    std::lock_guard<std::mutex> lk(g_dev_mu[dev]);
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob.data());
    if (mode == kModeMpdp && h->tree_mode == 0u && n <= 30 && gpuqo_b200_persistent != 0 && !profile) {
        auto &be = g_batch[dev];
        if (!be) be.reset(new BatchEngine());
        if (int rc = be->init(err)) return rc;
        if (be->persistent_ready()) {
            std::vector<const std::vector<uint32_t> *> wave(1, &blob);
            std::vector<std::vector<TreeNode>> wout;
            std::vector<int> redo;
            EngineStats st;
            double ms = 0.0;
            if (int rc = be->run_wave(wave, wout, redo, st, ms, err)) return rc;
            if (redo.empty()) {
                nodes = std::move(wout[0]);
                stats.connected_sets += st.connected_sets;
                stats.filtered_subsets += st.filtered_subsets;
                stats.evaluated_pairs += st.evaluated_pairs;
                stats.memo_bytes = st.memo_bytes;
                stats.device_ms += st.device_ms;
                stats.kernel_launches += st.kernel_launches;
                stats.barrier_timeouts += st.barrier_timeouts;
                return 0;
            }
        }
    }
    auto &eng = g_engines[dev];
    if (!eng) eng.reset(new Engine());
    return eng->run(blob, n, mode, ccc, profile, nodes, stats, err);
}

int engine_time_resident(const std::vector<uint32_t> &blob, int n, DpMode mode, bool ccc, int warmup, int iters,
                         bool flush_l2, double &ms_per_iter, std::vector<TreeNode> &nodes, EngineStats &stats,
                         std::string &err) {
    if (n < 1 || n > 31) {
        err = "exact DP supports 1..31 relations";
        return GPUQO_B200_ERR_TOO_LARGE;
    }
    int dev = 0;
    if (int rc = current_device(dev, err)) return rc;
    std::lock_guard<std::mutex> lk(g_dev_mu[dev]);
    // the same routing as engine_run: graphs with cycles as one-query waves
    const DevHeader *h = reinterpret_cast<const DevHeader *>(blob.data());
    if (mode == kModeMpdp && h->tree_mode == 0u && n <= 30 && gpuqo_b200_persistent != 0 && iters > 0) {
        auto &be = g_batch[dev];
        if (!be) be.reset(new BatchEngine());
        if (int rc = be->init(err)) return rc;
        if (be->persistent_ready()) {
            std::vector<const std::vector<uint32_t> *> wave(1, &blob);
            const size_t flush_bytes = 256u << 20;
            if (flush_l2 && !be->flush) CK(cudaMalloc(&be->flush, flush_bytes));
            double total = 0.0;
            bool ok = true;
            for (int i = 0; ok && i < warmup + iters; i++) {
                if (flush_l2) CK(cudaMemsetAsync(be->flush, i & 0xFF, flush_bytes, be->stream));
                std::vector<std::vector<TreeNode>> wout;
                std::vector<int> redo;
                EngineStats st;
                double ms = 0.0;
                if (int rc = be->run_wave(wave, wout, redo, st, ms, err)) return rc;
                ok = redo.empty();
                if (i >= warmup) total += ms;
                if (ok && i == warmup + iters - 1) {
                    nodes = std::move(wout[0]);
                    stats.connected_sets += st.connected_sets;
                    stats.filtered_subsets += st.filtered_subsets;
                    stats.evaluated_pairs += st.evaluated_pairs;
                    stats.memo_bytes = st.memo_bytes;
                    stats.kernel_launches += st.kernel_launches;
                }
                stats.barrier_timeouts += st.barrier_timeouts;
            }
            if (ok) {
                ms_per_iter = total / iters;
                stats.device_ms += ms_per_iter;
                return 0;
            }
        }
    }
    auto &eng = g_engines[dev];
    if (!eng) eng.reset(new Engine());
    return eng->time_resident(blob, n, mode, ccc, warmup, iters, flush_l2, ms_per_iter, nodes, stats, err);
}

// ---------------------------------------------------------------------------
// Autotuner.  On tree-shaped blobs of growing size (the host passes synthetic
// stars) it times k_dp_tree<2>, <3> and <4> device-resident, and one batch
// wave holding about 2^24 connected sets against single launches, then
// installs in the device's tuning record the three crossovers: up to which
// count of connected sets per level the 2-blocks variant beats the 3-blocks
// one at that size and every smaller one, from which count per level the
// 4-blocks variant wins at that size and every larger one (per level: the
// variants trade latency against throughput within a level, and the count per
// level carries over from stars to deeper trees, where the total does not),
// and from which total count a single launch beats its share of a wave.
// ---------------------------------------------------------------------------
static double crossover(const std::vector<double> &sets, const std::vector<bool> &wins) {
    size_t i = wins.size();
    while (i > 0 && wins[i - 1]) i--;
    if (i == wins.size()) return 1e30;     // never wins
    if (i == 0) return 0.0;                // wins from the smallest size on
    return std::sqrt(sets[i - 1] * sets[i]);
}

// the same from below: the largest count up to which `wins` holds at every size
static double crossover_below(const std::vector<double> &sets, const std::vector<bool> &wins) {
    size_t i = 0;
    while (i < wins.size() && wins[i]) i++;
    if (i == 0) return 0.0;                // loses at the smallest size
    if (i == wins.size()) return 1e30;     // wins at every size
    return std::sqrt(sets[i - 1] * sets[i]);
}

int engine_autotune(const std::vector<std::vector<uint32_t>> &blobs, double &single_narrow_level_sets,
                    double &single_wide_level_sets, double &batch_single_sets, std::string &err) {
    int dev = 0;
    if (int rc = current_device(dev, err)) return rc;
    std::lock_guard<std::mutex> lk(g_dev_mu[dev]);
    auto &eng = g_engines[dev];
    if (!eng) eng.reset(new Engine());
    auto &be = g_batch[dev];
    if (!be) be.reset(new BatchEngine());
    if (int rc = be->init(err)) return rc;
    std::vector<double> sets, level_sets;
    std::vector<bool> narrow_wins, wide_wins, single_wins;
    for (const auto &blob : blobs) {
        const DevHeader *h = reinterpret_cast<const DevHeader *>(blob.data());
        if (!h->tree_mode) continue;
        double t[3] = {0.0, 0.0, 0.0};   // k_dp_tree<2>, <3>, <4>
        for (int v = 0; v < 3; v++) {
            eng->force_minb = 2 + v;
            std::vector<TreeNode> nodes;
            EngineStats st;
            const int rc = eng->time_resident(blob, h->n, kModeMpdp, true, 1, 3, false, t[v], nodes, st, err);
            eng->force_minb = 0;
            if (rc) return rc;
        }
        const double cs = tree_connected_sets(h);
        const int m = (int)std::min(256.0, std::max(2.0, std::ceil(double(1u << 24) / cs)));
        std::vector<const std::vector<uint32_t> *> wave(m, &blob);
        double wms = 0.0;
        for (int rep = 0; rep < 2; rep++) {   // the first wave sizes the arena
            std::vector<std::vector<TreeNode>> wout;
            std::vector<int> redo;
            EngineStats st;
            if (int rc = be->run_wave(wave, wout, redo, st, wms, err)) return rc;
        }
        sets.push_back(cs);
        level_sets.push_back(cs / h->n);
        // each variant against the best of the other two, so that the
        // crossovers give the fastest of the three at every measured size
        narrow_wins.push_back(t[0] < std::min(t[1], t[2]));
        wide_wins.push_back(t[2] < std::min(t[0], t[1]));
        single_wins.push_back(std::min(t[0], std::min(t[1], t[2])) < wms / m);
    }
    single_narrow_level_sets = crossover_below(level_sets, narrow_wins);
    single_wide_level_sets = crossover(level_sets, wide_wins);
    batch_single_sets = crossover(sets, single_wins);
    Tuning &tu = g_tuning[dev];
    tu.single_narrow_level_sets = single_narrow_level_sets;
    tu.single_wide_level_sets = single_wide_level_sets;
    tu.batch_single_sets = batch_single_sets;
    tu.tuned = true;
    return 0;
}

void engine_set_tuning(double single_narrow_level_sets, double single_wide_level_sets, double batch_single_sets,
                       bool tuned) {
    int dev = 0;
    std::string err;
    if (current_device(dev, err)) dev = 0;   // no device yet: the record of device 0
    std::lock_guard<std::mutex> lk(g_dev_mu[dev]);
    Tuning &tu = g_tuning[dev];
    tu.single_narrow_level_sets = single_narrow_level_sets;
    tu.single_wide_level_sets = single_wide_level_sets;
    tu.batch_single_sets = batch_single_sets;
    tu.tuned = tuned;
}

int engine_reset_persistent() {
    int dev = 0;
    std::string err;
    if (current_device(dev, err)) return 0;
    std::lock_guard<std::mutex> lk(g_dev_mu[dev]);
    int cleared = 0;
    if (g_engines[dev] && g_engines[dev]->barrier_timed_out) {
        g_engines[dev]->barrier_timed_out = false;
        cleared++;
    }
    if (g_batch[dev] && g_batch[dev]->barrier_timed_out) {
        g_batch[dev]->barrier_timed_out = false;
        cleared++;
    }
    if (wide_reset_persistent(dev)) cleared++;
    return cleared;
}

void engine_get_tuning(double &single_narrow_level_sets, double &single_wide_level_sets, double &batch_single_sets, bool &tuned) {
    int dev = 0;
    std::string err;
    if (current_device(dev, err)) dev = 0;
    std::lock_guard<std::mutex> lk(g_dev_mu[dev]);
    const Tuning &tu = g_tuning[dev];
    single_narrow_level_sets = tu.single_narrow_level_sets;
    single_wide_level_sets = tu.single_wide_level_sets;
    batch_single_sets = tu.batch_single_sets;
    tuned = tu.tuned;
}

}  // namespace gqb
