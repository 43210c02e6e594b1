"""The work that users of this library have it do, as measurable cases.

A case is a dict of plain values.  ``prepare`` builds what a planner holds before the call (GpuqoPlannerInfoC
structures in host memory: the entry points take host structures, as the Postgres planner glue passes them), ``run``
makes one pass through the public entry points and returns the plans, ``work`` says what the pass cannot do without
and ``exact`` the optimum's cost in 64 bits, from a restatement of the cost model in numpy.

Kinds of case
  plan    one query through gpuqo_run with an exact algorithm (what a backend does per query)
  batch   many independent queries through gpuqo_b200_run_batch
  idp     one large query through gpuqo_run with gpuqo_idp_n_iters set (IDP2 or UnionDP over MPDP)
  served  a burst of large queries through the planner service
"""
import ctypes
import math
import os
import struct
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "postgres-gpuqo_b200"))

from gpuqo_b200 import capi, lib, query  # noqa: E402

IDP_TYPES = {"idp2": capi.GPUQO_IDP2, "union": capi.GPUQO_UNION}


# ----------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------
def _plan(name, shape, n, algorithm, stats=False, extra=0.0):
    return {"name": name, "kind": "plan", "shape": shape, "n": n, "algorithm": algorithm, "stats": stats,
            "extra": extra}


def listed():
    return [
        # a handful of joined tables, the commonest query there is: the fixed cost of a call
        _plan("star6-mpdp", "star", 6, "mpdp"),
        # plain DPsub on a dozen tables (the reference's default when gpuqo_dpsub_bicc is off)
        _plan("star12-dpsub", "star", 12, "dpsub"),
        # the headline query: MPDP of a 25-relation snowflake
        _plan("snowflake25-mpdp", "snowflake", 25, "mpdp"),
        # the largest single star that plans within a millisecond: throughput of one query
        _plan("star22-mpdp", "star", 22, "mpdp"),
        # many narrow levels on a graph with a cycle
        _plan("cycle30-dpsub", "key_cycle", 30, "dpsub"),
        # every subset of a clique is a valid side: 3^n pairs, the largest exact search
        _plan("clique18-dpsub", "clique", 18, "dpsub"),
        # a general join graph with column statistics and indexes (what ANALYZEd tables give)
        _plan("random16-stats-mpdp", "random", 16, "mpdp", stats=True, extra=0.12),
        # more relations than a dense memo holds: rings joined by paths on the sparse memo
        _plan("ringpath42-mpdp", "ring_path", 42, "mpdp"),
        # many small queries planned together
        {"name": "batch512-n8to16", "kind": "batch", "queries": 512, "nmin": 8, "nmax": 16},
        # fewer and larger ones
        {"name": "batch96-n10to20", "kind": "batch", "queries": 96, "nmin": 10, "nmax": 20},
        # one query far beyond exact search
        {"name": "idp2-snowflake200", "kind": "idp", "n": 200, "idp": "idp2", "k": 25},
        # a burst of such queries to the planner service
        {"name": "served16-union", "kind": "served", "requests": 16, "nmin": 30, "nmax": 150, "idp": "union", "k": 25},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    stats = rng.random() < 0.3
    what = rng.choice(["tree", "tree", "tree", "cycle", "clique", "random", "sparse", "batch", "idp", "served"])
    if what == "tree":
        shape = rng.choice(["star", "snowflake", "snowflake", "key_chain"])
        n = rng.randint(5, {"star": 20, "snowflake": 26, "key_chain": 30}[shape])
        c = _plan("", shape, n, rng.choice(["mpdp", "mpdp", "dpsub"]), stats)
    elif what == "cycle":
        c = _plan("", "key_cycle", rng.randint(6, 30), rng.choice(["mpdp", "dpsub"]), stats)
    elif what == "clique":
        c = _plan("", "clique", rng.randint(6, 17), "dpsub", False)
    elif what == "random":
        c = _plan("", "random", rng.randint(7, 16), rng.choice(["mpdp", "dpsub"]), stats,
                  round(rng.uniform(0.02, 0.12), 3))
    elif what == "sparse":
        shape = rng.choice(["key_chain", "key_cycle", "ring_path", "lollipop"])
        n = rng.randint(33, {"key_chain": 63, "key_cycle": 60, "ring_path": 42, "lollipop": 60}[shape])
        c = _plan("", shape, n, "mpdp", stats)
    elif what == "batch":
        nmax = rng.randint(11, 18)
        c = {"kind": "batch", "queries": log(64, 512 if nmax < 17 else 128), "nmin": rng.randint(6, 10), "nmax": nmax}
    elif what == "idp":
        c = {"kind": "idp", "n": log(35, 200), "idp": rng.choice(["idp2", "union"]), "k": rng.choice([15, 20, 25])}
    else:
        c = {"kind": "served", "requests": rng.randint(4, 16), "nmin": 30, "nmax": rng.randint(40, 150),
             "idp": "union", "k": rng.choice([15, 20, 25])}
    c.pop("name", None)
    return c


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _query(case, seed):
    if case["shape"] == "random":
        return query.random_graph(case["n"], seed, extra_edge_p=case["extra"], rich=case["stats"])
    return query.make(case["shape"], case["n"], seed, rich=case["stats"])


def _queries(case, seed):
    """The queries of a case.  The case alone decides how many there are, of which shape and size; the seed decides
    their graphs, row counts and selectivities."""
    if case["kind"] == "batch":
        # the shares of query.batch_mix: 40 % stars, 40 % snowflakes, 10 % chains, 10 % cycles
        rng = np.random.default_rng([case["queries"], case["nmin"], case["nmax"]])
        shapes = rng.choice(["star", "snowflake", "chain", "cycle"], case["queries"], p=[0.4, 0.4, 0.1, 0.1])
        ns = rng.integers(case["nmin"], case["nmax"] + 1, case["queries"])
        return [query.make(str(s), int(n), seed * 100003 + i) for i, (s, n) in enumerate(zip(shapes, ns))]
    if case["kind"] == "idp":
        return [query.snowflake(case["n"], seed)]
    if case["kind"] == "served":
        rng = np.random.default_rng([case["requests"], case["nmin"], case["nmax"]])
        ns = np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"] + 1), case["requests"])).astype(int)
        return [query.snowflake(int(n), seed * 1009 + i) for i, n in enumerate(ns)]
    return [_query(case, seed)]


_server = None    # the planner service, kept for the process as a planning process keeps it


def prepare(case, seed):
    global _server
    library = lib.load()
    built = [capi.PlannerInfoBuilder(q) for q in _queries(case, seed)]
    state = {"kind": case["kind"], "lib": library, "built": built,
             "infos": (ctypes.POINTER(capi.GpuqoPlannerInfoC) * len(built))(*[b.pointer() for b in built]),
             "trees": (ctypes.POINTER(capi.QueryTreeC) * len(built))(),
             "gucs": [(ctypes.c_bool.in_dll(library, "gpuqo_dpsub_bicc_enable"), case.get("algorithm") != "dpsub"),
                      (ctypes.c_int.in_dll(library, "gpuqo_idp_n_iters"), case.get("k", 0)),
                      (ctypes.c_int.in_dll(library, "gpuqo_idp_type"), IDP_TYPES[case.get("idp", "idp2")])]}
    if case["kind"] == "served" and _server is None:
        _server = lib.Server(max_inflight=16)
    return state


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------
# QueryTreeC: id, rows, startup, total, width, left, right
_NODE = struct.Struct("<Q3fi2Q")
# this process's memory, from one page on, as bytes and as 64-bit words
_BASE = 4096
_MEM = (ctypes.c_char * (1 << 46)).from_address(_BASE)
_WORDS = np.frombuffer((ctypes.c_uint64 * (1 << 43)).from_address(_BASE), dtype=np.uint64)


def _relation(bitmapset):
    """The relation of a leaf's one-bit Bitmapset (relation i is bit i + 1)."""
    words = ctypes.c_int.from_address(bitmapset).value
    for w in range(words):
        bits = ctypes.c_uint64.from_address(bitmapset + 8 + 8 * w).value
        if bits:
            return 64 * w + bits.bit_length() - 2
    return -1


def _read_plan(root):
    """A QueryTreeC as arrays, level by level from the root: per node its two children (-1 at a leaf), its relation
    (-1 at a join, whose id is the union of its children's), width, rows and costs."""
    todo = [root]
    rel, left, right, width, rows, startup, total = [], [], [], [], [], [], []
    for node in todo:
        ident, r, s, t, w, lp, rp = _NODE.unpack_from(_MEM, node - _BASE)
        rows.append(r)
        startup.append(s)
        total.append(t)
        width.append(w)
        if lp:
            rel.append(-1)
            left.append(len(todo))
            right.append(len(todo) + 1)
            todo.append(lp)
            todo.append(rp)
        else:
            rel.append(_relation(ident))
            left.append(-1)
            right.append(-1)
    return {"nodes": np.array([rel, left, right, width], dtype=np.int64), "rows": np.array(rows, dtype=np.float32),
            "startup": np.array(startup, dtype=np.float32), "total": np.array(total, dtype=np.float32),
            "cost": np.array(total[:1], dtype=np.float32)}


def _read_plans(roots):
    """Many plans as the same arrays at once (the roots come first, node numbers are over all plans)."""
    at = np.array(roots, dtype=np.uint64)
    parts, count = [], 0
    while at.size:
        word = ((at - np.uint64(_BASE)) >> np.uint64(3)).astype(np.int64)
        fields = _WORDS[word[:, None] + np.arange(5)]
        join = fields[:, 3] != 0
        child = count + at.size + 2 * (np.cumsum(join) - 1)
        ident = ((fields[:, 0] - np.uint64(_BASE)) >> np.uint64(3)).astype(np.int64)
        bits = np.zeros(at.size, dtype=np.int64)
        set_words = (_WORDS[ident] & np.uint64(0xFFFFFFFF)).astype(np.int64)
        for w in range(int(set_words[~join].max(initial=0))):
            one = np.where(~join & (set_words > w), _WORDS[np.where(set_words > w, ident + 1 + w, ident)], np.uint64(0))
            bits = np.where(one != 0, 64 * w + np.log2(np.maximum(one, np.uint64(1)).astype(np.float64)).astype(
                np.int64) - 1, bits)
        parts.append((np.where(join, -1, bits), np.where(join, child, -1), np.where(join, child + 1, -1),
                      (fields[:, 2] >> np.uint64(32)).astype(np.uint32).view(np.int32).astype(np.int64),
                      fields[:, 1:3].copy().view(np.float32)))
        count += at.size
        at = fields[join][:, 3:5].reshape(-1)
    value = np.concatenate([p[4] for p in parts])
    return {"nodes": np.stack([np.concatenate([p[i] for p in parts]) for i in range(4)]),
            "rows": np.ascontiguousarray(value[:, 0]), "startup": np.ascontiguousarray(value[:, 1]),
            "total": np.ascontiguousarray(value[:, 2]), "cost": np.ascontiguousarray(value[:len(roots), 2])}


def _address(pointer):
    return ctypes.cast(pointer, ctypes.c_void_p).value


def run(state):
    library = state["lib"]
    for guc, value in state["gucs"]:
        guc.value = value
    kind = state["kind"]
    if kind in ("plan", "idp"):
        tree = _address(library.gpuqo_run(capi.GPUQO_DPSUB, state["infos"][0]))
        if not tree:
            raise RuntimeError("gpuqo_run: error %d" % library.gpuqo_b200_last_error())
        plan = _read_plan(tree)
        library.gpuqo_b200_free_query_tree(tree)
        return plan
    n = len(state["built"])
    if kind == "batch":
        status = library.gpuqo_b200_run_batch(capi.GPUQO_DPSUB, state["infos"], n, state["trees"])
        if status:
            raise RuntimeError("gpuqo_b200_run_batch: %d" % status)
        trees = np.ctypeslib.as_array(ctypes.cast(state["trees"], ctypes.POINTER(ctypes.c_uint64)), (n,)).tolist()
    else:
        tickets = [_server.submit_built(b) for b in state["built"]]
        trees = []
        for ticket in tickets:
            status, tree, _ = _server.wait_raw(ticket)
            if status:
                raise RuntimeError("gpuqo_b200_server_wait: %d" % status)
            trees.append(_address(tree))
    plans = _read_plans(trees)
    for tree in trees:
        library.gpuqo_b200_free_query_tree(tree)
    return plans


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
# float operations of one costed pair: row estimate, nested loop and hash join, comparison
PAIR_FLOPS = 50


def _tree_pairs(q):
    """Ordered splits of all connected subsets of a tree: 2 (|S| - 1) for each (polynomials in |S| per subtree)."""
    order, parent = [0], {0: -1}
    for u in order:
        for v in q.edges[u]:
            if v not in parent:
                parent[v] = u
                order.append(v)
    poly, total = {}, np.zeros(q.n + 1)
    for u in reversed(order):
        p = np.array([0.0, 1.0])
        for v in q.edges[u]:
            if parent.get(v) == u:
                p = np.convolve(p, np.concatenate(([1.0], poly[v][1:])))
        poly[u] = p
        total[:len(p)] += p
    return float(sum(total[k] * 2 * (k - 1) for k in range(2, q.n + 1)))


def _connected_table(q):
    """connected[mask] for all subsets (up to 18 relations)."""
    sets = np.arange(1 << q.n, dtype=np.uint32)
    reach = sets & (~sets + np.uint32(1))
    adj = [sum(1 << v for v in q.edges[u]) for u in range(q.n)]
    while True:
        grown = reach.copy()
        for u in range(q.n):
            grown |= np.where((reach >> np.uint32(u)) & np.uint32(1), np.uint32(adj[u]), np.uint32(0))
        grown &= sets
        if np.array_equal(grown, reach):
            return (reach == sets) & (sets != 0)
        reach = grown


def _pairs(q):
    """Ordered pairs (L, R) of disjoint connected sets with a connected union, all of which exact search costs."""
    n, edges = q.n, sum(len(e) for e in q.edges) // 2
    if edges == n - 1:
        return _tree_pairs(q)
    if edges == n * (n - 1) // 2:
        return 3.0 ** n - 2.0 ** (n + 1) + 1
    if edges == n and all(len(e) == 2 for e in q.edges):   # a cycle: its arcs, and the splits of the whole
        return float(sum(n * 2 * (k - 1) for k in range(2, n)) + n * (n - 1))
    if n <= 18:   # ranked subset convolution of the connected sets with themselves
        conn = _connected_table(q)
        size = np.array([bin(i).count("1") for i in range(1 << n)])
        ranked = np.zeros((n + 1, 1 << n))
        for k in range(1, n + 1):
            ranked[k] = conn & (size == k)
        for b in range(n):
            v = ranked.reshape(n + 1, -1, 2, 1 << b)
            v[:, :, 1] += v[:, :, 0]
        total = 0.0
        for k in range(2, n + 1):
            conv = sum(ranked[i] * ranked[k - i] for i in range(1, k))
            for b in range(n):
                v = conv.reshape(-1, 2, 1 << b)
                v[:, 1] -= v[:, 0]
            total += float(conv[conn & (size == k)].sum())
        return total
    # larger sparse graphs: at least one split per spanning-tree edge of each connected set
    adj = np.array([sum(1 << v for v in q.edges[u]) for u in range(n)], dtype=np.uint64)
    level, total = np.uint64(1) << np.arange(n, dtype=np.uint64), 0.0
    for k in range(2, n + 1):
        grown = []
        for v in range(n):
            bit = np.uint64(1 << v)
            grown.append(level[((level & bit) == 0) & ((level & adj[v]) != 0)] | bit)
        level = np.unique(np.concatenate(grown))
        total += 2.0 * (k - 1) * level.size
    return total


def work(case):
    """Bytes: the planner infos in, the plans out.  Flops: the cost model once per pair that the search must cost
    (of a representative query where the seed decides the graph)."""
    if case["kind"] == "plan":
        q = _query(case, 0)
        relations, classes, pairs = q.n, len(q.eq_classes), _pairs(q)
    elif case["kind"] == "batch":
        relations, classes, pairs = 0, 0, 0.0
        for q in _queries(case, 0):
            relations += q.n
            classes += len(q.eq_classes)
            pairs += _pairs(q)
    else:
        # IDP2 solves one exact problem of k relations per k - 1 relations it joins; UnionDP partitions of up to k
        # relations, most of them smaller
        sizes = [q.n for q in _queries(case, 0)]
        relations, classes = sum(sizes), sum(sizes) - len(sizes)
        k = case["k"]
        of = _tree_pairs(query.snowflake(k if case["idp"] == "idp2" else max(k // 2, 2), 0))
        pairs = sum(math.ceil((n - 1) / (k - 1)) for n in sizes) * of
    # BaseRelationC and its id and edge sets, EqClassInfo with two members, QueryTreeC with its id
    return {"bytes": relations * 72.0 + classes * 176.0 + (2 * relations) * 56.0, "flops": pairs * PAIR_FLOPS}


# ----------------------------------------------------------------------------
# the optimum's cost in 64 bits
# ----------------------------------------------------------------------------
def _hash_size(tuples, width):
    """Buckets and batches of a hash table over `tuples` rows (work_mem 4 MB, pointers of 8 bytes)."""
    tupsize = 32 + ((width + 7) // 8) * 8
    allowed = 4096 * 1024
    table = np.where(allowed * 2 // 100 >= tupsize + 84, allowed - allowed * 2 // 100, allowed)
    pointers = 2.0 ** math.floor(math.log2(allowed / 8))
    buckets = 2.0 ** np.ceil(np.log2(np.maximum(np.minimum(np.ceil(tuples), pointers), 1024)))
    many = tuples * tupsize + 8 * buckets > table
    few = np.minimum(2.0 ** np.ceil(np.log2(table // (tupsize + 8))), pointers)
    batches = np.minimum(np.ceil(tuples * tupsize / (table - 8 * few)), pointers)
    batches = np.maximum(2.0 ** np.ceil(np.log2(np.maximum(batches, 1))), 2)
    return np.where(many, few, buckets), np.where(many, batches, 1.0)


def _clamp(rows):
    return np.where(rows <= 1, 1.0, np.rint(rows))


def _nestloop(o, i_rows, i_startup, i_total, unique, indexed, frac, inner_rows, per_tuple):
    run_inner = i_total - i_startup
    cost = o[2] - o[1] + np.where(o[0] > 1, (o[0] - 1) * i_startup, 0)
    plain = cost + run_inner + np.where(o[0] > 1, (o[0] - 1) * run_inner, 0)
    matched = np.rint(o[0] * frac)
    rest = o[0] - matched
    scan = 2 / (inner_rows + 1)
    tuples = matched * i_rows * scan
    if indexed:
        uniq = cost + run_inner * scan + np.where(matched > 1, (matched - 1) * run_inner * scan, 0)
        uniq = uniq + rest * run_inner / i_rows
    else:
        tuples = tuples + rest * i_rows
        m2, r2 = np.where(rest >= 1, matched, matched - 1), np.where(rest >= 1, rest - 1, rest)
        uniq = cost + run_inner + np.where(m2 > 0, m2 * run_inner * scan, 0) + np.where(r2 > 0, r2 * run_inner, 0)
    tuples = np.where(unique, tuples, o[0] * i_rows)
    startup = i_startup + o[1]
    return startup, startup + np.where(unique, uniq, plain) + (0.01 + per_tuple) * tuples


def _join(q, left, right, lv, rv, width):
    """Rows, startup and total cost of joining the sets `left` (outer) and `right` (inner) with values lv, rv."""
    single = (right & (right - 1)) == 0
    sel, quals = np.ones(left.size), np.zeros(left.size)
    unique, indexes = np.zeros(left.size, dtype=bool), []
    bucket, mcv = np.ones(left.size), np.ones(left.size)
    buckets, batches = _hash_size(rv[0], width[1])
    virtual = buckets * batches
    for ec in q.eq_classes:
        a, b = ec.members
        for x, y, jx, jy in ((a, b, 0, 1), (b, a, 1, 0)):   # x on the outer side, y on the inner
            hit = (((left >> x) & 1) & ((right >> y) & 1)).astype(bool)
            if not hit.any():
                continue
            s = ec.sels[0]
            if y in ec.fks[jx]:
                s = 1 / max(1.0, q.tuples[y])
            elif x in ec.fks[jy]:
                s = 1 / max(1.0, q.tuples[x])
            sel = np.where(hit, sel * s, sel)
            quals = quals + hit
            v = ec.vars[jy]
            distinct = -v.stadistinct * q.tuples[y] if v.stadistinct < 0 else v.stadistinct
            if distinct <= 0:
                size = np.full(left.size, 0.1)
            else:
                average = (1 - v.stanullfrac) / distinct
                if q.tuples[y] > 0:
                    distinct = float(_clamp(distinct * (q.rows[y] / q.tuples[y])))
                size = np.where(distinct > virtual, 1 / virtual, 1 / distinct)
                if average > 0 and v.mcvfreq > average:
                    size = size * (v.mcvfreq / average)
                size = np.clip(size, 1e-6, 1)
            bucket = np.where(hit, np.minimum(bucket, size), bucket)
            mcv = np.where(hit, np.minimum(mcv, v.mcvfreq), mcv)
            if v.index_available:
                indexes.append((hit & single, v))
                if v.index_unique:
                    unique = unique | (hit & single)
    product = sel * lv[0] * rv[0]
    rows = np.where(product > 1, np.floor(product + 0.5), 1.0)
    frac = rows / (lv[0] * rv[0])
    per_tuple = 0.0025 * quals
    startup, total = _nestloop(lv, rv[0], rv[1], rv[2], unique, False, frac, rv[0], per_tuple)
    # hash join
    hs = lv[1] + rv[2] + (0.0025 * quals + 0.01) * rv[0]
    hr = lv[2] - lv[1] + 0.0025 * quals * lv[0]
    pages = [np.ceil(v[0] * (((w + 7) // 8) * 8 + 24) / 8192) for v, w in zip((lv, rv), width)]
    hs = hs + np.where(batches > 1, pages[1], 0)
    hr = hr + np.where(batches > 1, pages[1] + 2 * pages[0], 0)
    hs = hs + np.where(_clamp(rv[0] * mcv) * (((width[1] + 7) // 8) * 8 + 24) > 4096 * 1024, 1e10, 0)
    matched = np.rint(lv[0] * frac)
    hr = hr + np.where(unique,
                       per_tuple * matched * _clamp(rv[0] * bucket * (2 / (rv[0] + 1))) * 0.5
                       + per_tuple * (lv[0] - matched) * _clamp(rv[0] / virtual) * 0.05 + 0.01 * matched,
                       per_tuple * lv[0] * _clamp(rv[0] * bucket) * 0.5 + 0.01 * rows)
    better = hs + hr < total
    startup, total = np.where(better, hs, startup), np.where(better, hs + hr, total)
    for hit, v in indexes:
        s, t = _nestloop(lv, v.index_rows, v.index_startup, v.index_total, unique, True, frac, rv[0], per_tuple)
        better = hit & (t < total)
        startup, total = np.where(better, s, startup), np.where(better, t, total)
    return rows, startup, total


def exact(case, seed):
    if case["kind"] != "plan":
        return None    # IDP is a heuristic whose choices follow 32-bit costs; a batch is too many searches
    q = _query(case, seed)
    if any(len(ec.members) != 2 for ec in q.eq_classes):
        return None
    n = q.n
    tree = sum(len(e) for e in q.edges) // 2 == n - 1
    adj = np.array([sum(1 << v for v in q.edges[u]) for u in range(n)], dtype=np.int64)
    levels = [np.left_shift(np.int64(1), np.arange(n, dtype=np.int64))]
    count = n
    for k in range(2, n + 1):
        grown = [levels[-1][((levels[-1] >> v) & 1 == 0) & ((levels[-1] & adj[v]) != 0)] | np.int64(1 << v)
                 for v in range(n)]
        levels.append(np.unique(np.concatenate(grown)))
        count += levels[-1].size
        if count > (300000 if tree else 4000):
            return None    # more than some seconds of numpy
    rows = [np.array(q.rows, dtype=np.float64)]
    startup = [np.array(q.startup, dtype=np.float64)]
    total = [np.array(q.total, dtype=np.float64)]
    width = [np.array(q.width, dtype=np.int64)]
    side = []    # a tree's edges as the relations on one end's side
    if tree:
        for a in range(n):
            for b in q.edges[a]:
                if a < b:
                    seen, todo = {a, b}, [a]
                    for u in todo:
                        todo += [v for v in q.edges[u] if v not in seen]
                        seen.update(q.edges[u])
                    side.append((a, b, np.int64(sum(1 << u for u in todo))))

    size_of = np.frompyfunc(lambda m: bin(m).count("1"), 1, 1)
    for k in range(2, n + 1):
        sets = levels[k - 1]
        best = [np.ones(sets.size), np.zeros(sets.size), np.full(sets.size, np.inf)]
        wide = np.zeros(sets.size, dtype=np.int64)
        parts = []
        if tree:
            for a, b, of in side:
                at = np.nonzero(((sets >> a) & 1) & ((sets >> b) & 1))[0]
                for mask in (of, ~of):
                    parts.append((at, sets[at] & mask))
        else:
            for i in range(1, k):
                one, two = levels[i - 1], levels[k - i - 1]
                for first in range(0, one.size, 256):
                    x = one[first:first + 256]
                    far, near = x[:, None] & two[None, :], np.zeros((x.size, two.size), dtype=bool)
                    for u in range(n):
                        near |= (((x >> u) & 1).astype(bool))[:, None] & ((two & adj[u]) != 0)[None, :]
                    xi, yi = np.nonzero((far == 0) & near)
                    parts.append((np.searchsorted(sets, x[xi] | two[yi]), x[xi]))
        for at, left in parts:
            if not at.size:
                continue
            right = sets[at] ^ left
            values, widths = [], []
            for part in (left, right):
                v, w = np.empty((3, at.size)), np.empty(at.size, dtype=np.int64)
                sizes = size_of(part).astype(int)
                for s in np.unique(sizes):
                    m = sizes == s
                    j = np.searchsorted(levels[s - 1], part[m])
                    v[0, m], v[1, m], v[2, m], w[m] = rows[s - 1][j], startup[s - 1][j], total[s - 1][j], width[s - 1][j]
                values.append(v)
                widths.append(w)
            got = _join(q, left, right, values[0], values[1], widths)
            order = np.argsort(got[2], kind="stable")
            first = order[np.unique(at[order], return_index=True)[1]]
            first = first[got[2][first] < best[2][at[first]]]
            for b, g in zip(best, got):
                b[at[first]] = g[first]
            wide[at] = widths[0] + widths[1]
        rows.append(best[0])
        startup.append(best[1])
        total.append(best[2])
        width.append(wide)
    return {"nodes": None, "rows": None, "startup": None, "total": None, "cost": total[n - 1].copy()}
