"""GPU: plain DPsub on cliques at the limits of its dense kernel: the largest
query whose sets are all one warp's and the smallest with shared sets, run in
turn (shares leave their arrays as the next query expects them), and queries
just below, at and beyond its 256 classes, against the oracle."""
import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query
from gpuqo_b200.query import EqClass, VarInfo

pytestmark = pytest.mark.gpu


def _run(q):
    got = lib.run(q, capi.GPUQO_DPSUB, bicc=False)
    assert got.error == 0 and same_tree(got.tree, harness.run_port(q, 3)[0])


def test_whole_and_shared_sets_in_turn():
    for n in (11, 12, 11, 13, 12, 5, 12):
        _run(query.clique(n, 20 + n))


def _classes(q, count):
    """a query with more classes on its edges, `count` in all"""
    first = list(q.eq_classes)
    for i in range(count - len(first)):
        q.eq_classes.append(EqClass(list(first[i % len(first)].members), [query.f32(0.5 + 0.001 * i)], [[], []],
                                    [VarInfo(), VarInfo()]))
    return q


@pytest.mark.parametrize("n,count", [(13, 234), (12, 255), (12, 256), (12, 257)])
def test_many_classes(n, count):
    _run(_classes(query.clique(n, n), count))
