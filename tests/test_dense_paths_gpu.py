"""GPU: plain DPsub over all subsets of dense graphs (the straight-line kernel
of plain classes, whole sets per warp and shares of a set) against the oracle,
at the sizes where its dispatch divides: one and two words of classes per
relation, sets of 11 and 12 relations, graphs at half of all edges and just
below, and the queries that it leaves to the general kernels (statistics, an
edge without a class, a class of three, keys both ways)."""
import numpy as np
import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query
from gpuqo_b200.query import EqClass, VarInfo

pytestmark = pytest.mark.gpu


def _dense(n, missing, seed, kind="plain"):
    pairs = [(a, b) for a in range(n) for b in range(a + 1, n)]
    rng = np.random.default_rng([n, missing, seed])
    drop = set(rng.permutation(len(pairs))[:missing].tolist())
    pairs = [p for i, p in enumerate(pairs) if i not in drop]
    if kind == "equal":
        rows, edges = [1000.0] * n, [(a, b, 0.5, None) for a, b in pairs]
    elif kind == "overflow":
        rows, edges = [1e20] * n, [(a, b, 1.0, None) for a, b in pairs]
    else:
        rows = np.exp(rng.uniform(5, 14, n))
        edges = [(a, b, float(np.exp(rng.uniform(-9, -2))), "a" if rng.uniform() < 0.3 else None) for a, b in pairs]
    q = query._assemble(f"dense{n}", n, rows, [int(w) for w in rng.integers(4, 65, n)], edges, rng,
                        rich=(kind == "stats"))
    if kind == "no_class":
        del q.eq_classes[2]
    elif kind == "class_of_3":
        q.eq_classes.append(EqClass([0, 1, 2], [query.f32(0.1)] * 3, [[], [], []], [VarInfo()] * 3))
    elif kind == "keys_both_ways":
        a, b = q.eq_classes[0].members
        q.eq_classes[0].fks = [[b], [a]]
    return q


CASES = [(2, 0, "plain"), (3, 0, "plain"), (6, 7, "plain"), (6, 8, "plain"), (11, 0, "plain"), (12, 0, "plain"),
         (13, 5, "plain"), (13, 39, "plain"), (14, 0, "plain"), (12, 3, "equal"), (12, 3, "overflow"), (4, 0, "overflow"),
         (12, 0, "stats"), (12, 0, "no_class"), (12, 0, "class_of_3"), (12, 0, "keys_both_ways")]


@pytest.mark.parametrize("n,missing,kind", CASES)
def test_dense_dpsub(n, missing, kind):
    q = _dense(n, missing, 3, kind)
    want = harness.run_port(q, 3)[0]
    for ccc in (True, False):
        got = lib.run(q, capi.GPUQO_DPSUB, bicc=False, ccc=ccc)
        assert got.error == 0 and same_tree(got.tree, want)
    # the same candidates with the block enumeration off and on
    lib.set_gucs(gpuqo_dpsub_csg_enable=False)
    try:
        assert same_tree(lib.run(q, capi.GPUQO_DPSUB, bicc=False, ccc=True).tree, want)
    finally:
        lib.set_gucs(gpuqo_dpsub_csg_enable=True)


def test_dense_dpsub_two_words():
    """17 relations: 136 classes, eight words per relation, shares of a set;
    the optimum is MPDP's."""
    q = query.clique(17, 5)
    a = lib.run(q, capi.GPUQO_DPSUB, bicc=False)
    b = lib.run(q, capi.GPUQO_DPSUB, bicc=True)
    assert a.error == 0 and b.error == 0
    assert a.stats["evaluated_pairs"] == b.stats["evaluated_pairs"] == 3 ** 17 - 2 ** 18 + 1
    assert a.tree[3] == b.tree[3] and a.tree[1] == b.tree[1]
