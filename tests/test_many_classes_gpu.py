"""GPU: planner infos of some 70 and 90 KB (850 and 1,100 classes), beyond the
shared memory that a launch has without being allowed it, larger and smaller in
turn, in the persistent kernels and by the launches per level, against the
oracle."""
import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query
from gpuqo_b200.query import EqClass, VarInfo

pytestmark = pytest.mark.gpu


def _with_classes(q, count):
    first = list(q.eq_classes)
    for i in range(count - len(first)):
        q.eq_classes.append(EqClass(list(first[i % len(first)].members), [query.f32(0.9)], [[], []], [VarInfo()] * 2))
    return q


@pytest.mark.parametrize("persistent", [1, 0])
@pytest.mark.parametrize("shape", ["star", "cycle", "clique"])
def test_many_classes(shape, persistent):
    L = lib.load()
    capi.set_int(L, "gpuqo_b200_persistent", persistent)
    try:
        for count in (1100, 850, 1100, 40, 1100):
            q = _with_classes(query.make(shape, 8, 3), count)
            for alg in (5, 3):
                got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
                assert got.error == 0 and same_tree(got.tree, harness.run_port(q, alg)[0])
    finally:
        capi.set_int(L, "gpuqo_b200_persistent", 1)
