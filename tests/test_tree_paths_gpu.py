"""GPU: where the evaluation of tree-shaped queries divides - the straight-line
cost of plain trees, the edge-class pass and the general pass, the 32-bit and
the 64-bit hash table size, packed and plain memo widths - each side against
the oracle, bit for bit, one query per side of each division."""
import ctypes as C

import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query
from gpuqo_b200.query import EqClass, VarInfo

pytestmark = pytest.mark.gpu


def _two_classes(q):
    """a second class on every third edge, with its own key"""
    for k, ec in enumerate(list(q.eq_classes)):
        if k % 3 == 0:
            a, b = ec.members
            q.eq_classes.append(EqClass([a, b], [query.f32(0.37)], [[], [a]], [VarInfo(), VarInfo()]))
    return q


def _no_class(q):
    """an edge without a class (a cross join)"""
    del q.eq_classes[1]
    return q


def _class_off_edges(q):
    """a class between two relations that no edge joins"""
    a, b = next((a, b) for a in range(q.n) for b in range(a + 1, q.n) if b not in q.edges[a])
    q.eq_classes.append(EqClass([a, b], [query.f32(0.5)], [[], []], [VarInfo(), VarInfo()]))
    return q


def _widths(q, w):
    q.width = [w + (i % 5) for i in range(q.n)]
    return q


QUERIES = {
    "plain": lambda: query.snowflake(13, 31),
    "two_classes": lambda: _two_classes(query.snowflake(13, 32)),
    "no_class": lambda: _no_class(query.snowflake(12, 33)),
    "class_off_edges": lambda: _class_off_edges(query.snowflake(12, 34)),
    "stats": lambda: query.snowflake(12, 35, rich=True),
    "wide_rows": lambda: _widths(query.star(11, 36), 150000),        # packed widths, rows near work_mem
    "width_sum_2^21": lambda: _widths(query.star(11, 37), 200000),   # widths sum beyond the packed range
    "equal_costs": lambda: query.random_graph(13, 38, extra_edge_p=0.0, equal=True),
    "overflow": lambda: query.chain(26, 39),                         # costs reach inf and NaN
    "two": lambda: query.star(2, 40),
}
# work_mem in kB around the bounds of the 32-bit hash table size (4 MB, 1 GB)
# and of one row; join methods off
SETTINGS = {"work_mem=64": {"work_mem": 64}, "work_mem=4095": {"work_mem": 4095}, "work_mem=4096": {"work_mem": 4096},
            "work_mem=1048575": {"work_mem": 1048575}, "work_mem=1048576": {"work_mem": 1048576},
            "nestloop_off": {"enable_nestloop": False}, "hashjoin_off": {"enable_hashjoin": False}}


def _set(settings):
    saved = []
    for library in (lib.load(), harness.load_port()):
        for name, value in settings.items():
            var = (C.c_bool if isinstance(value, bool) else C.c_int).in_dll(library, name)
            saved.append((var, var.value))
            var.value = value
    return saved


@pytest.mark.parametrize("setting", sorted(SETTINGS))
@pytest.mark.parametrize("name", sorted(QUERIES))
def test_tree_evaluation(name, setting):
    q = QUERIES[name]()
    saved = _set(SETTINGS[setting])
    try:
        for alg in ((5, 3) if q.n <= 13 else (5,)):
            got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
            assert got.error == 0
            if alg == 5:   # two relations are a complete graph, which plain DPsub enumerates by subsets
                assert got.stats["kernel_launches"] == 1
            want = harness.run_port(q, alg)[0]
            assert same_tree(got.tree, want)
            # the same through a batch wave (its planner infos stay in global memory)
            trees, rc = lib.run_batch([q, query.star(3, 1), q], capi.GPUQO_DPSUB, bicc=(alg == 5))
            assert rc == 0 and same_tree(trees[0], want) and same_tree(trees[2], want)
    finally:
        for var, value in saved:
            var.value = value
