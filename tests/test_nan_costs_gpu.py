"""GPU: trees whose row estimates overflow, so that candidates have infinite and
NaN costs (the reference keeps a NaN that is a set's first candidate and skips
it elsewhere), in narrow and wide levels, block order and plain DPsub's, with
and without statistics, alone and in a wave, against the oracle."""
import numpy as np
import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query

pytestmark = pytest.mark.gpu


def _overflowing(kind, n, rich):
    """large relations, hardly filtered: a few of them exceed a float"""
    rng = np.random.default_rng([n, len(kind)])
    pairs = {"star": [(0, i) for i in range(1, n)], "chain": [(i, i + 1) for i in range(n - 1)],
             "random": [(int(rng.integers(0, i)), i) for i in range(1, n)]}[kind]
    rows = [float(x) for x in rng.choice([1e7, 1e9, 1e12], n)]
    edges = [(a, b, float(rng.choice([0.5, 0.9])), None) for a, b in pairs]
    return query._assemble(f"overflow_{kind}{n}", n, rows, [8] * n, edges, rng, perm=rng.permutation(n), rich=rich)


QUERIES = {f"{kind}{n}{'_stats' if rich else ''}": (lambda k=kind, m=n, r=rich: _overflowing(k, m, r))
           for kind, sizes in (("star", (7, 13)), ("chain", (9, 20, 30)), ("random", (8, 13, 14)))
           for n in sizes for rich in (False, True)}
QUERIES["no_class"] = lambda: _without_a_class(_overflowing("random", 12, False))


def _without_a_class(q):
    del q.eq_classes[2]
    return q


@pytest.mark.parametrize("name", sorted(QUERIES))
def test_nan_costs(name):
    q = QUERIES[name]()
    for alg in (5, 3) if q.n <= 14 else (5,):
        want = harness.run_port(q, alg)[0]
        assert not np.isfinite(want[3])
        got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
        assert got.error == 0 and same_tree(got.tree, want)
        trees, rc = lib.run_batch([q, query.star(9, 1), q], capi.GPUQO_DPSUB, bicc=(alg == 5))
        assert rc == 0 and same_tree(trees[0], want) and same_tree(trees[2], want)


def test_time_with_nan_costs():
    """An overflowing chain against one of the same sets and splits without
    overflow: 1.73 times when every lane searched all splits of its set for
    the first candidate."""
    ms = [lib.time_resident(q, capi.GPUQO_DPSUB, bicc=True, warmup=3, iters=20)[1]
          for q in (query.key_chain(31, 1, rich=True), query.chain(31, 1, rich=True))]
    assert ms[1] < 1.5 * ms[0]
