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
// The splits come in another order than the reference's, whose index decides
// between equal costs and for a NaN: such sets are left to the block search
// (cactus_set returns false).
#pragma once

#include "dp_cactus_table.h"
#include "dp_device.cuh"

namespace gqb {

// One warp's scratch: per block the first split, the piece's first walk
// position and its relations
struct CactusScratch {
    uint16_t off[66];
    uint8_t start[64], size[64];
};

template <class M> __device__ __forceinline__ int cactus_popc(M x) { return sizeof(M) == 8 ? __popcll(x) : __popc((uint32_t)x); }

// the splits of S per block; returns their total
template <class M>
__device__ __forceinline__ uint32_t cactus_pieces(M S, const CactusView &v, CactusScratch &sc) {
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
__device__ __forceinline__ M cactus_side(M S, const CactusView &v, const CactusScratch &sc, uint32_t c, uint64_t &match) {
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
__device__ __forceinline__ void cactus_update(CactusBest<M> &best, M L, float rows, float startup, float total) {
    if (__builtin_expect(isnan(total), 0)) {
        best.nan = true;
        return;
    }
    const uint32_t ord = ord_float(total);
    if (ord == best.ord) best.tie = ord;
    if (ord < best.ord) {
        best.ord = ord;
        best.left = L;
        best.rows = rows;
        best.startup = startup;
    }
}

// A connected set by one warp: load(L) gives a side's memo entry, general(L,
// l, r, match, lr, rl) costs both orientations where plain_mirror does not
// apply, write(rows, startup, total, width, left) stores the winner (one
// lane).  False, and nothing written: equal lowest costs or a NaN.
template <class M, class Load, class General, class Write>
__device__ __forceinline__ bool cactus_set(M S, const CactusView &v, CactusScratch &sc, const PlainParams &pp, Load load,
                                           General general, Write write, uint32_t &pairs) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t W = cactus_pieces<M>(S, v, sc);
    CactusBest<M> best;
    best.ord = 0xFFFFFFFFu;
    best.tie = 0u;
    best.left = 0;
    best.rows = best.startup = 0.0f;
    best.nan = false;
    int width = 0;
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
        cactus_update<M>(best, L, lr.rows, lr.startup, lr.total);
        cactus_update<M>(best, R, rl.rows, rl.startup, rl.total);
    }
    const uint32_t ord = __reduce_min_sync(0xFFFFFFFFu, best.ord);
    const uint32_t win = __ballot_sync(0xFFFFFFFFu, best.ord == ord && ord != 0xFFFFFFFFu);
    if (__popc(win) != 1 || __any_sync(0xFFFFFFFFu, best.nan || (best.ord == ord && best.tie == ord))) return false;
    if ((win >> lane) & 1u)
        // the inverse of ord_float (a total is never -0: its startup cost starts from +0)
        write(best.rows, best.startup, __uint_as_float((ord & 0x80000000u) ? ord ^ 0x80000000u : ~ord), width, best.left);
    if (lane == 0u) pairs += 2u * W;
    return true;
}

}  // namespace gqb
