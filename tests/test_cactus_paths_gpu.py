"""GPU: cactus graphs (every block a bridge or a cycle) on the sparse memo's
persistent kernel - one ring up to 63 relations, rings around the 32-relation
word, triangles, rings sharing relations, statistics, equal and overflowing
costs, more than 64 classes, classes off the edges, arrays that have to grow -
against the oracle or, above its reach, the per-level launches."""
import numpy as np
import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query
from gpuqo_b200.query import EqClass, VarInfo

pytestmark = pytest.mark.gpu


def _ring(rels):
    return [(rels[i], rels[(i + 1) % len(rels)]) for i in range(len(rels))]


GRAPHS = {
    "ring63": (63, _ring(list(range(63)))),
    "ring32": (32, _ring(list(range(32)))),
    "ring33_tail": (35, _ring(list(range(33))) + [(7, 33), (33, 34)]),
    "triangles": (21, [e for i in range(0, 20, 2) for e in _ring([i, i + 1, i + 2])]),
    "rings_at_one": (16, _ring([0, 1, 2, 3]) + _ring([0, 4, 5, 6, 7]) + _ring([0, 8, 9]) + [(9, 10), (10, 11)] +
                     _ring([11, 12, 13, 14, 15])),
    "ring_bridges": (36, _ring(list(range(6))) + [(i, i + 1) for i in range(5, 33)] + _ring([33, 34, 35])),
}
KINDS = ["plain", "stats", "equal", "overflow", "two_classes", "off_edge", "no_class"]


def _query(name, kind):
    n, pairs = GRAPHS[name]
    rng = np.random.default_rng([n, len(pairs), KINDS.index(kind)])
    if kind == "equal":
        rows, edges = [1000.0] * n, [(a, b, 0.001, None) for a, b in pairs]
    elif kind == "overflow":
        rows, edges = [1e9] * n, [(a, b, 0.5, None) for a, b in pairs]
    else:
        rows = np.exp(rng.uniform(5, 14, n))
        edges = [(a, b, 1.0 / query.f32(round(float(rows[b]))), "a") for a, b in pairs]
    q = query._assemble(name, n, rows, [int(w) for w in rng.integers(4, 65, n)], edges, rng, rich=(kind == "stats"))
    if kind == "two_classes":   # beyond 64 classes on the larger graphs, keys both ways
        for ec in list(q.eq_classes):
            a, b = ec.members
            q.eq_classes.append(EqClass([a, b], [query.f32(0.7)], [[b], [a]], [VarInfo(), VarInfo()]))
    elif kind == "off_edge":
        a, b = next((a, b) for a in range(n) for b in range(a + 1, n) if b not in q.edges[a])
        q.eq_classes.append(EqClass([a, b], [query.f32(0.6)], [[], []], [VarInfo()] * 2))
    elif kind == "no_class":
        del q.eq_classes[1]
    return q


@pytest.fixture
def knob():
    L = lib.load()
    yield lambda name, v: capi.set_int(L, name, v)
    capi.set_int(L, "gpuqo_b200_sparse_from_rels", 32)
    capi.set_int(L, "gpuqo_b200_sparse_host_list", 0)
    capi.set_int(L, "gpuqo_b200_persistent", 1)
    capi.set_int(L, "gpuqo_b200_barrier_poll_limit", 0)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_cactus_on_the_sparse_memo(name, kind, knob):
    q = _query(name, kind)
    knob("gpuqo_b200_sparse_from_rels", 2)
    for alg in (5, 3):
        got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
        assert got.error == 0 and got.stats["kernel_launches"] == 1
        knob("gpuqo_b200_persistent", 0)
        levels = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
        knob("gpuqo_b200_persistent", 1)
        assert levels.stats["kernel_launches"] > 1
        assert same_tree(got.tree, levels.tree)
        assert got.stats["connected_sets"] == levels.stats["connected_sets"]
        assert got.stats["evaluated_pairs"] == levels.stats["evaluated_pairs"]
        assert same_tree(got.tree, harness.run_port(q, alg)[0])


@pytest.mark.parametrize("room", [1, 100, 1000])
def test_arrays_grow(room, knob):
    """The launch ends at the level that outgrows its arrays and is repeated
    with larger ones (ring path of 40: 15 thousand sets)."""
    q = query.ring_path(40, 1)
    want = lib.run(q, capi.GPUQO_DPSUB, bicc=True)
    knob("gpuqo_b200_sparse_host_list", room)
    got = lib.run(q, capi.GPUQO_DPSUB, bicc=True)
    assert got.error == 0 and got.stats["kernel_launches"] > 1 and want.stats["kernel_launches"] == 1
    assert same_tree(got.tree, want.tree)


def test_barrier_timeout_takes_the_level_launches(knob):
    q = query.key_cycle(40, 2)
    want = lib.run(q, capi.GPUQO_DPSUB, bicc=True).tree
    knob("gpuqo_b200_barrier_poll_limit", 1)
    got = lib.run(q, capi.GPUQO_DPSUB, bicc=True)
    assert got.error == 0 and got.stats["barrier_timeouts"] == 1 and same_tree(got.tree, want)
    knob("gpuqo_b200_barrier_poll_limit", 0)
    again = lib.run(q, capi.GPUQO_DPSUB, bicc=True)
    assert again.stats["barrier_timeouts"] == 0 and again.stats["kernel_launches"] > 1
    assert lib.load().gpuqo_b200_reset_persistent() >= 1
    back = lib.run(q, capi.GPUQO_DPSUB, bicc=True)
    assert back.stats["kernel_launches"] == 1 and same_tree(back.tree, want)
