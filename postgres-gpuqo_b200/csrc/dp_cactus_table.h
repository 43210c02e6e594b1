// dp_cactus_table.h - the table of a cactus query graph (every biconnected
// block a bridge or a simple cycle): layout, and its construction on the host.
// dp_cactus.cuh has what it is for.
#pragma once

#include <cstdint>
#include <cstring>
#include <vector>

#include "dp_layout.h"

namespace gqb {

struct CactusHead {
    uint32_t n_blocks;            // the cycles first
    uint32_t n_cycles;
    uint32_t n_walk;              // walk entries, m + 1 per block
    uint32_t flags;               // kCactusEdges, kCactusPlain
    uint32_t n_sets;              // connected sets of the graph (all ones: 2^32 - 1 or more)
    uint32_t pad[3];
};
static_assert(sizeof(CactusHead) == 32, "CactusHead layout");
constexpr uint32_t kCactusEdges = 1u;   // two-member classes on edges only, at most 64
constexpr uint32_t kCactusPlain = 2u;   // ... all plain, a class on every edge (plain_mirror applies)

// one two-member class {x < y}: its selectivity with x's side outer and with
// y's (pair_sel), and x
struct CactusClass {
    float lo, hi;
    uint32_t x, pad;
};

// sections of the table, in 8-byte words after the head
struct CactusView {
    CactusHead h;
    const uint64_t *mask;         // [n_blocks] the block's relations
    const uint64_t *pre;          // [n_walk] union of the parts of the first i relations of the walk
    const uint64_t *cls;          // [n_walk] classes on the edge from walk position i to the next
    const PlainQuals *quals;      // [n_ec + 1] (kCactusEdges)
    const CactusClass *classes;   // [n_ec] (kCactusEdges)
    const uint32_t *meta;         // [n_blocks] first walk entry | m << 16
    const uint8_t *vert;          // [n_walk] relation at walk position i
};

GQB_HD inline CactusView cactus_view(const void *tab, int n_ec) {
    CactusView v;
    v.h = *reinterpret_cast<const CactusHead *>(tab);
    const uint64_t *p = reinterpret_cast<const uint64_t *>(tab) + 4;
    const uint32_t ec = (v.h.flags & kCactusEdges) ? (uint32_t)n_ec : 0u;
    v.quals = reinterpret_cast<const PlainQuals *>(p);
    p += 2u * (ec + 1u);
    v.classes = reinterpret_cast<const CactusClass *>(p);
    p += 2u * ec;
    v.mask = p;
    p += v.h.n_blocks;
    v.pre = p;
    p += v.h.n_walk;
    v.cls = p;
    p += v.h.n_walk;
    v.meta = reinterpret_cast<const uint32_t *>(p);
    p += (v.h.n_blocks + 1u) / 2u;
    v.vert = reinterpret_cast<const uint8_t *>(p);
    return v;
}

// Host: the table of a connected graph, empty when it is no cactus.  rel: the
// classes' member masks, sel: both orientations of each two-member class,
// plain: plain_mirror applies to the classes (kCactusPlain, if every edge has
// one); quals(i): PlainQuals of i quals.
template <class Quals>
inline std::vector<uint64_t> build_cactus(const std::vector<uint64_t> &adj, const std::vector<uint64_t> &rel,
                                          const std::vector<float> &sel, bool plain, Quals quals) {
    const int n = (int)adj.size(), n_ec = (int)rel.size();
    struct Block {
        std::vector<int> walk;
        uint64_t mask;
    };
    std::vector<Block> cycles, bridges;
    // Connected sets: f[v] of them lie in v's part of the block tree (rooted at
    // relation 0) and contain v; a block's children are complete when it is
    // emitted.  A set's topmost piece is one relation (f) or a run of two or
    // more children of a cycle.
    double f[64], sets = 0.0;
    for (int i = 0; i < n; i++) f[i] = 1.0;
    {
        // blocks of the graph (depth-first, a relation stack); recursion
        // unrolled: at most 63 relations
        int disc[64], low[64], stk[64], par[64], vst[64], sp = 0, vs = 0, t = 0;
        uint64_t todo[64];
        for (int i = 0; i < n; i++) disc[i] = -1;
        disc[0] = low[0] = t++;
        par[0] = -1;
        todo[0] = adj[0];
        stk[sp++] = 0;
        vst[vs++] = 0;
        while (sp) {
            const int u = stk[sp - 1];
            if (todo[u]) {
                const int v = __builtin_ctzll(todo[u]);
                todo[u] &= todo[u] - 1ull;
                if (disc[v] < 0) {
                    disc[v] = low[v] = t++;
                    par[v] = u;
                    todo[v] = adj[v];
                    stk[sp++] = v;
                    vst[vs++] = v;
                } else if (v != par[u] && disc[v] < low[u]) {
                    low[u] = disc[v];
                }
                continue;
            }
            sp--;
            const int p = par[u];
            if (p < 0) break;
            if (low[u] < low[p]) low[p] = low[u];
            if (low[u] < disc[p]) continue;
            Block b;
            b.mask = 1ull << p;
            int w;
            do {
                w = vst[--vs];
                b.mask |= 1ull << w;
            } while (w != u);
            int m = 0, ends = 0;
            for (uint64_t x = b.mask; x; x &= x - 1ull, m++) ends += __builtin_popcountll(adj[__builtin_ctzll(x)] & b.mask);
            if (m > 2 && ends != 2 * m) return {};
            // from the lowest relation towards its lower neighbour
            int v = __builtin_ctzll(b.mask), prev = 63 - __builtin_clzll(adj[v] & b.mask);
            for (int i = 0; i < m; i++) {
                b.walk.push_back(v);
                const uint64_t rest = adj[v] & b.mask & ~(1ull << prev);
                prev = v;
                if (m == 2) v = 63 - __builtin_clzll(b.mask);
                else v = __builtin_ctzll(rest);
            }
            int top = 0;
            while (b.walk[(size_t)top] != p) top++;
            std::vector<double> child;
            for (int i = 1; i < m; i++) child.push_back(f[b.walk[(size_t)((top + i) % m)]]);
            // runs from either side of the top relation, then the whole block
            double with = 0.0, left = 1.0, all = 1.0;
            for (double x : child) all *= x;
            for (int i = 0; i <= m - 2; i++) {
                double right = 1.0;
                for (int j = 0; i + j <= m - 2; j++) {
                    with += left * right;
                    right *= child[(size_t)(m - 2 - j)];
                }
                left *= child[(size_t)i];
            }
            with += all;
            for (int i = 0; i < m - 1; i++) {
                double run = child[(size_t)i];
                sets += run;
                for (int j = i + 1; j < m - 1; j++) sets += run *= child[(size_t)j];
            }
            f[p] *= with;
            (m > 2 ? cycles : bridges).push_back(std::move(b));
        }
        if (t != n) return {};
        sets += f[0];
    }
    std::vector<Block> blocks = std::move(cycles);
    CactusHead head{};
    head.n_cycles = (uint32_t)blocks.size();
    blocks.insert(blocks.end(), bridges.begin(), bridges.end());
    head.n_blocks = (uint32_t)blocks.size();
    for (const Block &b : blocks) head.n_walk += (uint32_t)b.walk.size() + 1u;
    bool edges = n_ec <= 64;
    for (int i = 0; edges && i < n_ec; i++) {
        if (__builtin_popcountll(rel[i]) != 2) edges = false;
        else if (!((adj[__builtin_ctzll(rel[i])] & rel[i]))) edges = false;
    }
    head.flags = edges ? kCactusEdges : 0u;
    head.n_sets = sets < 4294967295.0 ? (uint32_t)sets : 0xFFFFFFFFu;
    std::vector<uint64_t> tab(4u + (edges ? 4u * (uint32_t)n_ec + 2u : 2u) + head.n_blocks + 2u * head.n_walk +
                                  (head.n_blocks + 1u) / 2u + (head.n_walk + 32u + 7u) / 8u + 1u,
                              0ull);
    tab.resize((tab.size() + 1u) & ~(size_t)1);
    std::memcpy(tab.data(), &head, sizeof(head));
    CactusView v = cactus_view(tab.data(), n_ec);
    if (edges) {
        for (int i = 0; i <= n_ec; i++) const_cast<PlainQuals *>(v.quals)[i] = quals(i);
        for (int i = 0; i < n_ec; i++) {
            CactusClass &c = const_cast<CactusClass *>(v.classes)[i];
            c.lo = sel[2 * i];
            c.hi = sel[2 * i + 1];
            c.x = (uint32_t)__builtin_ctzll(rel[i]);
        }
    }
    uint32_t at = 0u;
    bool every_edge = true;
    for (uint32_t b = 0; b < head.n_blocks; b++) {
        const Block &B = blocks[b];
        const uint32_t m = (uint32_t)B.walk.size();
        const_cast<uint64_t *>(v.mask)[b] = B.mask;
        const_cast<uint32_t *>(v.meta)[b] = at | (m << 16);
        uint64_t acc = 0ull;
        for (uint32_t i = 0; i < m; i++) {
            const int w = B.walk[i], nx = B.walk[(i + 1u) % m];
            const_cast<uint8_t *>(v.vert)[at + i] = (uint8_t)w;
            const_cast<uint64_t *>(v.pre)[at + i] = acc;
            // what hangs off w without the block's other relations
            uint64_t part = 1ull << w, next = part;
            while (next) {
                const int y = __builtin_ctzll(next);
                next &= next - 1ull;
                const uint64_t fresh = adj[y] & ~part & ~B.mask;
                part |= fresh;
                next |= fresh;
            }
            acc |= part;
            uint64_t on = 0ull;
            const uint64_t ends = (1ull << w) | (1ull << nx);
            if (edges && (m > 2u || i == 0u)) {
                for (int e = 0; e < n_ec; e++)
                    if (rel[e] == ends) on |= 1ull << e;
                every_edge = every_edge && on != 0ull;
            }
            const_cast<uint64_t *>(v.cls)[at + i] = on;
        }
        const_cast<uint64_t *>(v.pre)[at + m] = acc;
        at += m + 1u;
    }
    if (edges && plain && every_edge) {
        head.flags |= kCactusPlain;
        std::memcpy(tab.data(), &head, sizeof(head));
    }
    return tab;
}

}  // namespace gqb
