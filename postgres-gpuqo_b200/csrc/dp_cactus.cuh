// dp_cactus.cuh - connected sets of cactus query graphs (every biconnected
// block is a bridge or a simple cycle), without a block search.
//
// A connected set S meets each block of the graph in one connected piece:
// nothing, a single relation, a path along the block, or the whole cycle.
// Its own blocks are the edges of those paths and the whole cycles, so its
// unordered splits are the cuts of every path (one less than its relations)
// and the arcs of every whole cycle of m relations (m (m - 1) / 2 of them up to
// complement), all of them valid.  For each block the graph's relations fall
// into one part per block relation (what hangs off it outside the block): the
// union of the parts along a piece of the block, cut with S, is a side.  The
// unions along each block's walk are tabulated once per query (host,
// build_cactus); a prefix of the walk is one 8-byte entry, any arc the
// exclusive or of two.  The classes that a cut matches are those on its one or
// two edges when every class sits on an edge.
//
// Between equal costs the reference's order decides.  Plain DPsub's is that of
// the subsets of S, so of the outer sides as integers.  The block enumeration's
// is not at hand here: sets with equal lowest costs, and with a NaN cost, get
// their blocks searched in the reference's order (cactus_order) and their
// splits costed once more, with indices.
#pragma once

#include "dp_cactus_table.h"
#include "dp_device.cuh"

namespace gqb {

// One warp's scratch: per block of the graph the first split, the piece's
// first walk position and its relations; then the set's own blocks in the
// reference's order and the search stack (cactus_order)
template <class M>
struct CactusScratch {
    static constexpr int kRels = (int)sizeof(M) * 8;
    M mask[kRels], st_desc[kRels], st_reach[kRels], st_rem[kRels], st_adj[kRels];
    uint64_t prefix[kRels];
    uint16_t off[kRels + 2];
    uint8_t start[kRels], size[kRels], st_u[kRels];
    uint32_t nb;
};

template <class M> __device__ __forceinline__ int cactus_popc(M x) { return sizeof(M) == 8 ? __popcll(x) : __popc((uint32_t)x); }
template <class M> __device__ __forceinline__ uint32_t cactus_low(M x) {
    return (uint32_t)((sizeof(M) == 8 ? __ffsll((long long)x) : __ffs((int)(uint32_t)x)) - 1);
}

// the splits of S per block; returns their total
template <class M>
__device__ __forceinline__ uint32_t cactus_pieces(M S, const CactusView &v, CactusScratch<M> &sc) {
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
    for (uint32_t b = 0; b < v.h.n_cycles; b++) {
        const uint32_t base = v.meta[b] & 0xFFFFu, m = v.meta[b] >> 16;
        uint64_t at = __ballot_sync(0xFFFFFFFFu, lane < m && ((S >> v.vert[base + lane]) & 1u));
        if (sizeof(M) == 8 && m > 32u)
            at |= (uint64_t)__ballot_sync(0xFFFFFFFFu, lane + 32u < m && ((S >> v.vert[base + lane + 32u]) & 1u)) << 32;
        // the walk positions in S are one run around the cycle: it starts
        // where the position before is not in S
        const uint64_t first = at & ~((at << 1) | (at >> (m - 1u)));
        if (lane == 0u) {
            sc.size[b] = (uint8_t)__popcll(at);
            sc.start[b] = (uint8_t)(first ? __ffsll((long long)first) - 1 : 0);
        }
    }
    __syncwarp();
    uint32_t total = 0u;
#pragma unroll
    for (uint32_t part = 0; part < (sizeof(M) == 8 ? 2u : 1u); part++) {
        const uint32_t b = lane + 32u * part;
        uint32_t cnt = 0u;
        if (b < v.h.n_cycles) {
            const uint32_t a = sc.size[b], m = v.meta[b] >> 16;
            cnt = a == m ? m * (m - 1u) / 2u : (a >= 2u ? a - 1u : 0u);
        } else if (b < v.h.n_blocks) {
            const M blk = (M)v.mask[b];
            cnt = (S & blk) == blk ? 1u : 0u;
        }
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= (uint32_t)o) incl += x;
        }
        if (b < v.h.n_blocks) sc.off[b] = (uint16_t)(total + incl - cnt);
        total += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    __syncwarp();
    return total;
}

// one side of split c of S and the classes on the cut edges
template <class M>
__device__ __forceinline__ M cactus_side(M S, const CactusView &v, const CactusScratch<M> &sc, uint32_t c, uint64_t &match) {
    // the last block whose first split is at most c (blocks without splits
    // share their successor's)
    uint32_t b = 0u;
#pragma unroll
    for (uint32_t step = sizeof(M) == 8 ? 32u : 16u; step >= 1u; step >>= 1)
        if (b + step < v.h.n_blocks && sc.off[b + step] <= c) b += step;
    const uint32_t j = c - sc.off[b], base = v.meta[b] & 0xFFFFu, m = v.meta[b] >> 16;
    const bool cycle = b < v.h.n_cycles, whole = cycle && sc.size[b] == m;
    // a whole cycle's arcs by length (m of each length below m / 2, m / 2 of
    // that length), otherwise the first j + 1 relations of the piece
    const uint32_t s = whole ? j % m : (cycle ? sc.start[b] : 0u);
    const uint32_t e = s + (whole ? j / m : j) + 1u;
    const uint64_t *pre = v.pre + base;
    const uint64_t u = e <= m ? (pre[e] ^ pre[s]) : ((pre[m] ^ pre[s]) | pre[e - m]);
    match = v.cls[base + (e - 1u < m ? e - 1u : e - 1u - m)];
    if (whole) match |= v.cls[base + (s ? s - 1u : m - 1u)];
    return S & (M)u;
}

// A lane's best side by cost alone; tie: two of its orientations share the
// cost best.ord had when the second came
template <class M>
struct CactusBest {
    uint32_t ord, tie;
    M left;
    float rows, startup;
    bool nan;
};

template <class M>
__device__ __forceinline__ void cactus_update(CactusBest<M> &best, M L, bool dpsub, float rows, float startup,
                                              float total) {
    if (__builtin_expect(isnan(total), 0)) {
        best.nan = true;
        return;
    }
    const uint32_t ord = ord_float(total);
    if (ord == best.ord && !dpsub) best.tie = ord;
    if (ord < best.ord || (dpsub && ord == best.ord && L < best.left)) {
        best.ord = ord;
        best.left = L;
        best.rows = rows;
        best.startup = startup;
    }
}

// The set's blocks in the reference's output order and the candidates ahead of
// each (2^m - 2 per block): depth-first from the lowest relation, neighbours in
// increasing order, by lane 0 with masks (as gen_blocks)
template <class M, class Adj>
__device__ __noinline__ void cactus_order(M S, const Adj *adj, CactusScratch<M> &sc) {
    if ((threadIdx.x & 31u) == 0u) {
        int sp = 0;
        uint32_t nb = 0u, u = cactus_low<M>(S);
        M desc = (M)1 << u, rem = desc, reach = (M)adj[u], visited = desc, anc = 0, a = reach & S;
        uint64_t ahead = 0ull;
        for (;;) {
            const M c = a & ~visited;
            if (c) {
                sc.st_u[sp] = (uint8_t)u;
                sc.st_desc[sp] = desc;
                sc.st_reach[sp] = reach;
                sc.st_rem[sp] = rem;
                sc.st_adj[sp] = a;
                sp++;
                anc |= (M)1 << u;
                u = cactus_low<M>(c);
                desc = rem = (M)1 << u;
                visited |= desc;
                reach = (M)adj[u];
                a = reach & S;
            } else {
                if (sp == 0) break;
                sp--;
                const uint32_t p = sc.st_u[sp];
                const M bit = (M)1 << p;
                M up = sc.st_rem[sp];
                anc &= ~bit;
                if ((reach & anc) == 0) {
                    sc.mask[nb] = rem | bit;
                    sc.prefix[nb] = ahead;
                    ahead += (1ull << cactus_popc<M>(rem | bit)) - 2ull;
                    nb++;
                } else {
                    up |= rem;
                }
                desc |= sc.st_desc[sp];
                reach |= sc.st_reach[sp];
                rem = up;
                a = sc.st_adj[sp];
                u = p;
            }
        }
        sc.nb = nb;
    }
    __syncwarp();
}

// the bits of x at the positions of mask, packed (x within mask)
template <class M>
__device__ __forceinline__ uint64_t cactus_pext(M x, M mask) {
    uint64_t r = 0ull;
    for (; x; x &= x - 1) r |= 1ull << cactus_popc<M>(mask & ((x & (~x + 1)) - 1));
    return r;
}

// the reference's index of the candidate with outer side L (after
// cactus_order), or its place in plain DPsub's order
template <class M>
__device__ __noinline__ uint64_t cactus_index(M S, const CactusScratch<M> &sc, M L, bool dpsub) {
    if (dpsub) return (uint64_t)L;
    const M R = S ^ L;
    uint32_t b = 0u;
    // the one block that the split cuts
    while (b + 1u < sc.nb && ((sc.mask[b] & L) == 0 || (sc.mask[b] & R) == 0)) b++;
    return sc.prefix[b] + cactus_pext<M>(L & sc.mask[b], sc.mask[b]) - 1ull;
}

// A connected set by one warp: load(L) gives a side's memo entry, general(L,
// l, r, match, lr, rl) costs both orientations where plain_mirror does not
// apply, write(rows, startup, total, width word, left) stores the winner (one
// lane).
template <class M, class Adj, class Load, class General, class Write>
__device__ __forceinline__ void cactus_set(M S, const CactusView &v, const DevHeader &h, const Adj *adj,
                                           CactusScratch<M> &sc, bool dpsub, const PlainParams &pp, Load load, General general, Write write,
                                           uint32_t &pairs) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t W = cactus_pieces<M>(S, v, sc);
    CactusBest<M> best;
    best.ord = 0xFFFFFFFFu;
    best.tie = 0u;
    best.left = 0;
    best.rows = best.startup = 0.0f;
    best.nan = false;
    int width = 0;
    // second pass: the candidates' indices; the lowest one with the lowest
    // cost, the lowest one at all and whether its cost is a NaN
    bool exact = false, nans = false, first_nan = false;
    uint32_t ord = 0u;
    uint64_t best_p = ~0ull, first_p = ~0ull;
    float first_rows = 0.0f, first_startup = 0.0f, first_total = 0.0f;
    M first_left = 0;
    for (;;) {
        for (uint32_t c = lane; c < W; c += 32u) {
            uint64_t match;
            const M L = cactus_side<M>(S, v, sc, c, match), R = S ^ L;
            const float4 l = load(L), r = load(R);
            JoinCost lr, rl;
            if (v.h.flags & kCactusPlain) {
                float sel_l = 1.0f, sel_r = 1.0f;
                for (uint64_t x = match; x; x &= x - 1ull) {
                    const CactusClass k = v.classes[__ffsll((long long)x) - 1];
                    const bool lo = (L >> k.x) & 1u;
                    sel_l *= lo ? k.lo : k.hi;
                    sel_r *= lo ? k.hi : k.lo;
                }
                plain_mirror(pp, v.quals[__popcll(match)], sel_l, sel_r, l, r, lr, rl);
                width = (int)((__float_as_uint(l.w) & kWidthMask) + (__float_as_uint(r.w) & kWidthMask));
            } else {
                width = general(L, l, r, match, lr, rl);
            }
            if (!exact) {
                cactus_update<M>(best, L, dpsub, lr.rows, lr.startup, lr.total);
                cactus_update<M>(best, R, dpsub, rl.rows, rl.startup, rl.total);
                continue;
            }
#pragma unroll 1
            for (int side = 0; side < 2; side++) {
                const JoinCost &o = side ? rl : lr;
                const bool nan = isnan(o.total), lowest_cost = !nan && ord_float(o.total) == ord;
                if (!lowest_cost && !nans) continue;
                const M X = side ? R : L;
                const uint64_t p = cactus_index<M>(S, sc, X, dpsub);
                if (lowest_cost && p < best_p) {
                    best_p = p;
                    best.left = X;
                    best.rows = o.rows;
                    best.startup = o.startup;
                }
                if (p < first_p) {
                    first_p = p;
                    first_nan = nan;
                    first_left = X;
                    first_rows = o.rows;
                    first_startup = o.startup;
                    first_total = o.total;
                }
            }
        }
        if (exact) break;
        ord = __reduce_min_sync(0xFFFFFFFFu, best.ord);
        const uint32_t win = __ballot_sync(0xFFFFFFFFu, best.ord == ord && ord != 0xFFFFFFFFu);
        nans = __any_sync(0xFFFFFFFFu, best.nan);
        if (!nans && dpsub) {
            best_p = (win >> lane) & 1u ? (uint64_t)best.left : ~0ull;
            break;
        }
        if (!nans && __popc(win) == 1 && !__any_sync(0xFFFFFFFFu, best.ord == ord && best.tie == ord)) {
            best_p = (win >> lane) & 1u ? 0ull : ~0ull;
            break;
        }
        exact = true;
        if (!dpsub) cactus_order<M>(S, adj, sc);
    }
    auto least = [](uint64_t p) {
        const uint32_t hi = __reduce_min_sync(0xFFFFFFFFu, (uint32_t)(p >> 32));
        const uint32_t lo = __reduce_min_sync(0xFFFFFFFFu, (uint32_t)(p >> 32) == hi ? (uint32_t)p : 0xFFFFFFFFu);
        return ((uint64_t)hi << 32) | lo;
    };
    bool mine = best_p != ~0ull, kept = false;
    if (exact || dpsub) {   // every lane takes part in the reductions
        const uint64_t lowest_p = least(best_p);
        mine = mine && best_p == lowest_p;
        if (nans) {
            const uint64_t lowest_first = least(first_p);
            kept = first_nan && first_p == lowest_first;
            if (__any_sync(0xFFFFFFFFu, kept)) mine = false;
        }
    }
    auto word = [&](float rows) {
        return (v.h.flags & kCactusPlain) ? plain_width_word(h, rows, width) : memo_width_word(h, rows, width);
    };
    if (kept) write(first_rows, first_startup, first_total, word(first_rows), first_left);
    // the inverse of ord_float (a total is never -0: its startup cost starts from +0)
    if (mine)
        write(best.rows, best.startup, __uint_as_float((ord & 0x80000000u) ? ord ^ 0x80000000u : ~ord), word(best.rows),
              best.left);
    if (lane == 0u) pairs += 2u * W;
}

}  // namespace gqb
