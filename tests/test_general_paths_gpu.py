"""GPU: graphs with cycles at the sizes where their evaluation divides -
bridges, simple cycles (odd and even), blocks of 3 relations and more, several
blocks hanging off one another, sets just below and above the splits that one
warp takes alone, equal costs and overflowing (inf, NaN) ones - as one query
(MPDP, and plain DPsub where it takes the block enumeration) and as a batch
wave, against the oracle bit for bit."""
import numpy as np
import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query

pytestmark = pytest.mark.gpu


def _ring(first, m):
    return [(first + i, first + (i + 1) % m) for i in range(m)]


def _full(first, m):
    return [(first + i, first + j) for i in range(m) for j in range(i + 1, m)]


GRAPHS = {
    "triangle": (3, _full(0, 3)),
    "triangles": (9, [e for i in range(0, 8, 2) for e in _full(i, 3)]),
    "ring4": (4, _ring(0, 4)),
    "ring9_tail": (12, _ring(0, 9) + [(2, 9), (9, 10), (5, 11)]),
    "rings": (13, _ring(0, 5) + [(x + 4, y + 4) for x, y in _ring(0, 6)] + [(9, 10), (10, 11), (11, 12)]),
    "full8": (8, _full(0, 8)),                                   # 127 splits: one warp
    "full9": (9, _full(0, 9)),                                   # 255 splits: dealt out
    "full9_full6": (14, _full(0, 9) + [(x + 8, y + 8) for x, y in _full(0, 6)]),
    "ring_of_full": (12, _ring(0, 12) + _full(0, 5) + [(7, 9), (7, 10)]),
    "ring20": (20, _ring(0, 20)),
}


def _query(name, kind):
    n, pairs = GRAPHS[name]
    pairs = sorted(set((min(p), max(p)) for p in pairs))
    rng = np.random.default_rng([len(name), n, KINDS.index(kind)])
    if kind == "equal":
        rows, edges = [1000.0] * n, [(a, b, 0.01, None) for a, b in pairs]
    elif kind == "overflow":
        rows, edges = [1e12] * n, [(a, b, 0.5, None) for a, b in pairs]
    else:
        rows = np.exp(rng.uniform(5, 14, n))
        edges = [(a, b, 1.0 / query.f32(round(float(rows[b]))), "a") if rng.uniform() < 0.5 else
                 (a, b, float(np.exp(rng.uniform(-9, -2))), None) for a, b in pairs]
    q = query._assemble(name, n, rows, [int(w) for w in rng.integers(4, 65, n)], edges, rng,
                        rich=kind in ("stats", "stats_two_classes"))
    if kind in ("two_classes", "stats_two_classes"):   # beyond 32 classes on the larger graphs, keys both ways
        for ec in list(q.eq_classes):
            a, b = ec.members
            q.eq_classes.append(query.EqClass([a, b], [query.f32(0.7)], [[b], [a]], [query.VarInfo(), query.VarInfo()]))
    elif kind == "off_edge" and n > 3:
        far = [(a, b) for a in range(n) for b in range(a + 1, n) if b not in q.edges[a]]
        if far:
            q.eq_classes.append(query.EqClass(list(far[0]), [query.f32(0.6)], [[], []], [query.VarInfo()] * 2))
    elif kind == "no_class":
        del q.eq_classes[1]
    return q


KINDS = ["plain", "stats", "equal", "overflow", "two_classes", "stats_two_classes", "off_edge", "no_class"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_general_evaluation(name, kind):
    q = _query(name, kind)
    for alg in (5, 3):
        want = harness.run_port(q, alg)[0]
        got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
        assert got.error == 0 and same_tree(got.tree, want)
        trees, rc = lib.run_batch([q, query.cycle(5, 1), q], capi.GPUQO_DPSUB, bicc=(alg == 5))
        assert rc == 0 and same_tree(trees[0], want) and same_tree(trees[2], want)
