// dp_general.cuh - evaluation of connected sets of graphs with cycles: a
// warp's block search in shared memory, the unordered splits of every block,
// and the distribution of large sets over the grid.
//
// The reference costs, for every biconnected block b of a set S, every proper
// nonempty subset lb of b (gpuqo_cpu_dpsub_bicc.cu:46-236): L grows from lb
// and R from the rest, and the pair counts when they cover S.  A subset and
// its complement in the block give the same two sides in the two
// orientations, so here a candidate is an unordered split (half the subsets),
// tested once and costed in both orientations together.  Removing b leaves
// one part of S hanging off each of its relations; a side is the union of the
// parts of its relations, and it is valid when both sides are connected sets,
// which the enumeration's bitmap answers for every smaller set.
//
// A candidate's place in the reference's order is needed only where it
// decides: between equal costs and for NaN costs (the first candidate of a
// set, if its cost is NaN, is kept).  In block order it is the enumeration
// index, and the first candidate is always valid (a biconnected block without
// its lowest relation is connected); plain DPsub visits the subsets of S in
// increasing order, so there it is the outer side itself, and the first valid
// one is searched for.
#pragma once

#include "dp_cactus.cuh"
#include "dp_device.cuh"

namespace gqb {

// One warp's scratch (shared memory, 4 KB)
struct GenScratch {
    uint32_t mask[32];            // blocks in the reference's output order
    uint32_t sub[32];             // ... the relations below the block's child end in the search tree
    uint32_t prefix[33];          // ... candidates of the reference ahead of the block (2^m - 2 each)
    uint32_t half[33];            // ... unordered splits ahead of it
    // unions of the parts of a block's relations, 4 relations per group of 16
    // words (blocks of 3 and more relations that are no cycles: at most 14
    // groups for the 30 relations of this path, as triangles)
    uint32_t tab[16 * 16];
    uint32_t pre[64];             // cycle blocks: unions along the walk (sizes plus one, at most 48)
    uint32_t hang[32];            // relation and the parts below it outside its parent block
    alignas(16) uint32_t list[32];
    uint32_t st_desc[32], st_nb[32], st_rem[32], st_adj[32];   // search stack
    uint16_t off[32];             // first group in tab, or first word in pre
    uint8_t st_u[32];
    uint32_t nb, cyc;
    alignas(8) CactusScratch<uint32_t> cactus;
    alignas(8) uint32_t queue[64 * 2];       // valid splits waiting for a full warp: candidate, side
};

// Blocks of S in the reference's output order (depth-first from the lowest
// relation, neighbours in increasing order, a block emitted on the return
// over its first edge).  Lane 0 walks: a child closes a block when no relation
// of its subtree neighbours a proper ancestor of its parent, all masks, about
// 120 cycles per relation; the tables are filled by the whole warp.
__device__ __forceinline__ void gen_blocks(uint32_t S, const uint32_t *adj, GenScratch &ws) {
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
    ws.hang[lane] = 1u << lane;
    __syncwarp();
    if (lane == 0) {
        int sp = 0, nb = 0;
        uint32_t u = (uint32_t)lowest_idx(S), desc = 1u << u, rem = desc, reach = adj[u], visited = desc, anc = 0u;
        uint32_t a = reach & S;
        for (;;) {
            const uint32_t c = a & ~visited;
            if (c) {
                ws.st_u[sp] = (uint8_t)u;
                ws.st_desc[sp] = desc;
                ws.st_nb[sp] = reach;
                ws.st_rem[sp] = rem;
                ws.st_adj[sp] = a;
                sp++;
                anc |= 1u << u;
                u = (uint32_t)lowest_idx(c);
                desc = rem = 1u << u;
                visited |= desc;
                reach = adj[u];
                a = reach & S;
            } else {
                if (sp == 0) break;
                sp--;
                const uint32_t p = ws.st_u[sp], bit = 1u << p;
                uint32_t up = ws.st_rem[sp];
                anc &= ~bit;
                if ((reach & anc) == 0u) {
                    ws.mask[nb] = rem | bit;
                    ws.sub[nb] = desc;
                    nb++;
                    ws.hang[p] |= desc;
                } else {
                    up |= rem;
                }
                desc |= ws.st_desc[sp];
                reach |= ws.st_nb[sp];
                rem = up;
                a = ws.st_adj[sp];
                u = p;
            }
        }
        ws.nb = (uint32_t)nb;
    }
    __syncwarp();
    const uint32_t nb = ws.nb;
    // lane b: block b
    const uint32_t blk = lane < nb ? ws.mask[lane] : 0u, sub = lane < nb ? ws.sub[lane] : 0u;
    const uint32_t m = (uint32_t)popc(blk);
    bool cyc = m >= 4u;
    for (uint32_t x = blk; cyc && x; x &= x - 1u) cyc = popc(adj[lowest_idx(x)] & blk) == 2;
    const uint32_t full = m ? (1u << m) - 2u : 0u;
    const uint32_t half = m <= 2u ? (m ? 1u : 0u) : (cyc ? m * (m - 1u) / 2u : (1u << (m - 1u)) - 1u);
    const uint32_t words = m <= 2u ? 0u : (cyc ? (m + 1u) << 16 : (m + 3u) / 4u);
    uint32_t i_full = full, i_half = half, i_words = words;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t f = __shfl_up_sync(0xFFFFFFFFu, i_full, o), h = __shfl_up_sync(0xFFFFFFFFu, i_half, o),
                       w = __shfl_up_sync(0xFFFFFFFFu, i_words, o);
        if (lane >= (uint32_t)o) {
            i_full += f;
            i_half += h;
            i_words += w;
        }
    }
    const uint32_t off = cyc ? (i_words - words) >> 16 : (i_words - words) & 0xFFFFu;
    const uint32_t cycles = __ballot_sync(0xFFFFFFFFu, cyc), large = __ballot_sync(0xFFFFFFFFu, m >= 3u && !cyc);
    if (lane < nb) {
        ws.prefix[lane] = i_full - full;
        ws.half[lane] = i_half - half;
        ws.off[lane] = (uint16_t)off;
        if (lane == nb - 1u) {
            ws.prefix[nb] = i_full;
            ws.half[nb] = i_half;
        }
    }
    if (lane == 0) ws.cyc = cycles;
    if (cyc) {
        // from the block's lowest relation towards its lower neighbour
        int v = lowest_idx(blk), prev = 31 - __clz(adj[v] & blk);
        uint32_t acc = 0u;
        ws.pre[off] = 0u;
        for (uint32_t i = 1; i <= m; i++) {
            acc |= ((sub >> v) & 1u) ? ws.hang[v] : S & ~sub;
            ws.pre[off + i] = acc;
            const int nx = lowest_idx(adj[v] & blk & ~(1u << prev));
            prev = v;
            v = nx;
        }
    }
    for (uint32_t todo = large; todo; todo &= todo - 1u) {
        const uint32_t b = (uint32_t)lowest_idx(todo);
        const uint32_t bm = ws.mask[b], bs = ws.sub[b], size = (uint32_t)popc(bm), bit = 1u << lane;
        __syncwarp();
        if (bm & bit) ws.list[popc(bm & (bit - 1u))] = (bs & bit) ? ws.hang[lane] : S & ~bs;
        if (lane >= size) ws.list[lane] = 0u;
        __syncwarp();
        const uint32_t o = __shfl_sync(0xFFFFFFFFu, off, (int)b) * 16u;
        for (uint32_t x = lane; x < (size + 3u) / 4u * 16u; x += 32u) {
            const uint4 q = *reinterpret_cast<const uint4 *>(ws.list + ((x >> 4) << 2));
            ws.tab[o + x] = ((x & 1u) ? q.x : 0u) | ((x & 2u) ? q.y : 0u) | ((x & 4u) ? q.z : 0u) | ((x & 8u) ? q.w : 0u);
        }
    }
    __syncwarp();
}

// the block of split c
__device__ __forceinline__ uint32_t gen_block_of(const GenScratch &ws, const uint32_t *first, uint32_t c) {
    uint32_t b = 0u;
    const uint32_t nb = ws.nb;
    if (nb > 1u) {
#pragma unroll
        for (uint32_t step = 16u; step >= 1u; step >>= 1)
            if (b + step < nb && first[b + step] <= c) b += step;
    }
    return b;
}

// one side of the unordered split c of S; test: whether its two sides may be
// disconnected (blocks that are neither bridges nor cycles)
__device__ __forceinline__ uint32_t gen_side(uint32_t S, const GenScratch &ws, uint32_t c, bool &test) {
    const uint32_t b = gen_block_of(ws, ws.half, c);
    const uint32_t blk = ws.mask[b], j = c - ws.half[b], m = (uint32_t)popc(blk);
    test = false;
    if (m == 2u) {
        const uint32_t sub = ws.sub[b];
        return (lowest(blk) & sub) ? sub : S ^ sub;
    }
    if ((ws.cyc >> b) & 1u) {
        // arcs by length: m of each length below m / 2, m / 2 of that length
        const uint32_t *pre = ws.pre + ws.off[b];
        const uint32_t s = j % m, e = s + j / m + 1u;
        return e <= m ? (pre[e] ^ pre[s]) : ((pre[m] ^ pre[s]) | pre[e - m]);
    }
    test = true;
    const uint32_t *tab = ws.tab + ws.off[b] * 16u;
    uint32_t L = 0u;
    for (uint32_t x = j + 1u; x; x >>= 4, tab += 16) L |= tab[x & 15u];
    return L;
}

// the place of split c with L the outer side
__device__ __forceinline__ uint32_t gen_index(uint32_t S, const GenScratch &ws, uint32_t c, uint32_t L, uint32_t dpsub) {
    if (dpsub) return L;
    const uint32_t b = gen_block_of(ws, ws.half, c), blk = ws.mask[b];
    return ws.prefix[b] + pext32(L & blk, blk) - 1u;
}

// the outer side of the candidate at place p
__device__ __forceinline__ uint32_t gen_from_index(uint32_t S, const GenScratch &ws, uint32_t p, uint32_t dpsub) {
    if (dpsub) return p;
    const uint32_t b = gen_block_of(ws, ws.prefix, p), blk = ws.mask[b], bs = ws.sub[b];
    uint32_t L = 0u;
    for (uint32_t x = pdep32(p - ws.prefix[b] + 1u, blk); x; x &= x - 1u) {
        const int v = lowest_idx(x);
        L |= ((bs >> v) & 1u) ? ws.hang[v] : S & ~bs;
    }
    return L;
}

__device__ __forceinline__ bool seen_bit(const uint32_t *seen, uint32_t T) { return (seen[T >> 5] >> (T & 31u)) & 1u; }

// A lane's best orientation of a set (see TreeBest)
struct GenBest {
    uint32_t ord, c, left;
    float rows, startup;
    uint32_t nan_p;               // lowest place of a NaN candidate
    uint32_t pairs;

    __device__ __forceinline__ void init() {
        ord = 0xFFFFFFFFu;
        c = left = 0u;
        rows = startup = 0.0f;
        nan_p = 0xFFFFFFFFu;
        pairs = 0u;
    }
};

__device__ __forceinline__ void gen_update(GenBest &best, const DevHeader &h, const GenScratch &ws, uint32_t S,
                                           uint32_t c, uint32_t L, const RelVal &out) {
    const uint32_t ord = ord_float(out.total);
    bool take = ord < best.ord;
    if (__builtin_expect(ord == best.ord || isnan(out.total), 0)) {
        const uint32_t p = gen_index(S, ws, c, L, h.index_order);
        if (isnan(out.total)) {
            best.nan_p = min(best.nan_p, p);
            take = false;
        } else {
            take = p < gen_index(S, ws, best.c, best.left, h.index_order);
        }
    }
    if (take) {
        best.ord = ord;
        best.c = c;
        best.left = L;
        best.rows = out.rows;
        best.startup = out.startup;
    }
}

// both orientations of the valid split c = (L, S - L)
__device__ __forceinline__ void gen_cost(const DevInfoView &d, const GenScratch &ws, uint32_t S, uint32_t c, uint32_t L,
                                         const float4 *memo, GenBest &best, int &width) {
    const RelVal l = load_rel(memo, L, d.h->hz_packed), r = load_rel(memo, S ^ L, d.h->hz_packed);
    RelVal o0, o1;
    join_eval_mirror(d, L, l, S ^ L, r, o0, o1);
    width = o0.width;
    best.pairs += 2u;
    gen_update(best, *d.h, ws, S, c, L, o0);
    gen_update(best, *d.h, ws, S, c, S ^ L, o1);
}

// Splits [lo, hi) of S, the whole warp.  Valid splits wait in a queue until
// they fill the warp (most subsets of a sparse block are not connected).
__device__ __forceinline__ void gen_range(const DevInfoView &d, GenScratch &ws, uint32_t S, uint32_t lo, uint32_t hi,
                                          const float4 *memo, const uint32_t *seen, GenBest &best, int &width) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t queued = 0u;
    __syncwarp();
    for (uint32_t base = lo;;) {
        while (queued < 32u && base < hi) {
            const uint32_t c = base + lane;
            bool ok = c < hi, test = false;
            uint32_t L = 0u;
            if (ok) {
                L = gen_side(S, ws, c, test);
                if (test) ok = seen_bit(seen, L) && seen_bit(seen, S ^ L);
            }
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
            if (ok) {
                const uint32_t at = queued + (uint32_t)popc(m & ((1u << lane) - 1u));
                ws.queue[2u * at] = c;
                ws.queue[2u * at + 1u] = L;
            }
            queued += (uint32_t)popc(m);
            base += 32u;
        }
        if (queued == 0u) break;
        __syncwarp();
        const uint32_t take = min(queued, 32u);
        queued -= take;
        if (lane < take) {
            const uint2 e = *reinterpret_cast<const uint2 *>(ws.queue + 2u * (queued + lane));
            gen_cost(d, ws, S, e.x, e.y, memo, best, width);
        }
        __syncwarp();
    }
}

// place of the first valid candidate of S
__device__ __noinline__ uint32_t gen_first(uint32_t S, uint32_t dpsub, const uint32_t *seen) {
    if (!dpsub) return 0u;
    const uint32_t lane = threadIdx.x & 31u, total = (1u << popc(S)) - 2u;
    for (uint32_t base = 0u; base < total; base += 32u) {
        const uint32_t p = base + lane;
        const uint32_t L = p < total ? pdep32(p + 1u, S) : 0u;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, p < total && seen_bit(seen, L) && seen_bit(seen, S ^ L));
        if (m) return __shfl_sync(0xFFFFFFFFu, L, lowest_idx(m));
    }
    return 0xFFFFFFFFu;
}

// the memo entry of S from the candidate at place p (one lane writes)
__device__ __noinline__ void gen_write_index(const DevInfoView d, const GenScratch &ws, uint32_t S, uint32_t p,
                                             float4 *memo, uint32_t *memo_left) {
    if ((threadIdx.x & 31u) == 0u) {
        const uint32_t L = gen_from_index(S, ws, p, d.h->index_order);
        const RelVal l = load_rel(memo, L, d.h->hz_packed), r = load_rel(memo, S ^ L, d.h->hz_packed);
        const RelVal out = join_eval(d, L, l, S ^ L, r);
        memo[S] = make_float4(out.rows, out.startup, out.total,
                              __uint_as_float(memo_width_word(*d.h, out.rows, out.width)));
        memo_left[S] = L;
    }
    __syncwarp();
}

// lanes with the warp's lowest cost, the tie broken: the winner's lane (its
// place in p when ties were compared or want_p is set)
__device__ __forceinline__ bool gen_winner(const DevHeader &h, const GenScratch &ws, uint32_t S, const GenBest &best,
                                           bool want_p, uint32_t &ord, uint32_t &p) {
    ord = __reduce_min_sync(0xFFFFFFFFu, best.ord);
    bool win = best.ord == ord && ord != 0xFFFFFFFFu;
    const uint32_t tied = __ballot_sync(0xFFFFFFFFu, win);
    p = 0xFFFFFFFFu;
    if (want_p || popc(tied) > 1) {
        const uint32_t mine = win ? gen_index(S, ws, best.c, best.left, h.index_order) : 0xFFFFFFFFu;
        p = __reduce_min_sync(0xFFFFFFFFu, mine);
        win = win && mine == p;
    }
    return win;
}

// a set evaluated by its warp alone
__device__ __forceinline__ void gen_set(const DevInfoView &d, GenScratch &ws, uint32_t S, float4 *memo,
                                        uint32_t *memo_left, const uint32_t *seen, uint32_t &pairs) {
    GenBest best;
    best.init();
    int width = 0;
    gen_range(d, ws, S, 0u, ws.half[ws.nb], memo, seen, best, width);
    pairs += best.pairs;
    uint32_t ord, p;
    bool win = gen_winner(*d.h, ws, S, best, false, ord, p);
    if (__any_sync(0xFFFFFFFFu, best.nan_p != 0xFFFFFFFFu)) {
        const uint32_t nan_p = __reduce_min_sync(0xFFFFFFFFu, best.nan_p);
        if (nan_p == gen_first(S, d.h->index_order, seen)) {
            win = false;
            gen_write_index(d, ws, S, nan_p, memo, memo_left);
        }
    }
    if (win) {
        // the inverse of ord_float (a total is never -0: its startup cost starts from +0)
        const float total = __uint_as_float((ord & 0x80000000u) ? ord ^ 0x80000000u : ~ord);
        memo[S] = make_float4(best.rows, best.startup, total, __uint_as_float(memo_width_word(*d.h, best.rows, width)));
        memo_left[S] = best.left;
    }
}

// a set of a cactus graph (table cv), by its pieces
__device__ __forceinline__ void gen_cactus_set(const DevInfoView &d, const CactusView &cv, const PlainParams &pp,
                                               GenScratch &ws, uint32_t S, float4 *memo, uint32_t *memo_left,
                                               uint32_t &pairs) {
    const DevHeader &h = *d.h;
    cactus_set<uint32_t>(
        S, cv, h, h.adj, ws.cactus, h.index_order != 0u, pp, [&](uint32_t L) { return __ldcg(memo + L); },
        [&](uint32_t L, const float4 lv, const float4 rv, uint64_t match, JoinCost &lr, JoinCost &rl) {
            const RelVal l = unpack_rel(lv, h.hz_packed), r = unpack_rel(rv, h.hz_packed);
            RelVal o0, o1;
            if ((cv.h.flags & kCactusEdges) && h.n_ec <= 32)
                join_eval_mirror_w<1, true>(d, L, l, S ^ L, r, (uint32_t)match, o0, o1);
            else
                join_eval_mirror(d, L, l, S ^ L, r, o0, o1);
            lr.rows = o0.rows;
            lr.startup = o0.startup;
            lr.total = o0.total;
            rl.rows = o1.rows;
            rl.startup = o1.startup;
            rl.total = o1.total;
            return o0.width;
        },
        [&](float rows, float startup, float total, uint32_t word, uint32_t left) {
            memo[S] = make_float4(rows, startup, total, __uint_as_float(word));
            memo_left[S] = left;
        },
        pairs);
}

}  // namespace gqb
