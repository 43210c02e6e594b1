"""GPU: trees whose memo is beyond the caches (more used sectors than the L2
cache holds, or a span of more than 512 MB) are listed in another order: their
plans against the oracle or, above its reach, the per-level launches, which
list by themselves, and the time of a star far beyond L2 against one just
beyond it."""
import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query

pytestmark = pytest.mark.gpu


def _by_level(q, alg):
    L = lib.load()
    capi.set_int(L, "gpuqo_b200_persistent", 0)
    try:
        r = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
    finally:
        capi.set_int(L, "gpuqo_b200_persistent", 1)
    assert r.error == 0 and r.stats["kernel_launches"] > 1
    return r.tree


@pytest.mark.parametrize("alg", [5, 3])
def test_span_beyond_512_mb(alg):
    q = query.snowflake(26, 1)          # 1 GB of memo, 0.2 million connected sets
    got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
    assert got.error == 0 and got.stats["kernel_launches"] == 1
    assert same_tree(got.tree, harness.run_port(q, 5)[0] if alg == 5 else _by_level(q, alg))


# below and above the bounds: 2 and 8.4 million sets of plain trees and of ones
# with statistics, spans of 512 MB and 1 GB; equal costs; a chain whose costs
# overflow
@pytest.mark.parametrize("make", [
    lambda: query.star(22, 2), lambda: query.star(24, 2), lambda: query.star(24, 3, rich=True),
    lambda: query.snowflake(25, 4), lambda: query.snowflake(27, 5), lambda: query.snowflake(28, 6, rich=True),
    lambda: query.random_graph(26, 7, extra_edge_p=0.0, equal=True), lambda: query.chain(29, 8)])
@pytest.mark.parametrize("alg", [5, 3])
def test_orders_give_one_plan(make, alg):
    q = make()
    got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
    assert got.error == 0 and got.stats["kernel_launches"] == 1
    assert same_tree(got.tree, _by_level(q, alg))


def test_wave_beyond_512_mb():
    qs = [query.snowflake(25, 11), query.chain(25, 12), query.star(14, 13), query.snowflake(24, 14), query.star(2, 15)]
    trees, rc = lib.run_batch(qs, capi.GPUQO_DPSUB, bicc=True)
    assert rc == 0
    for q, tree in zip(qs, trees):
        assert same_tree(tree, lib.run(q, capi.GPUQO_DPSUB, bicc=True).tree)


def test_time_of_a_star_follows_its_pairs():
    """star-26 has 4.3 times the pairs of star-24.  Where every memo entry of
    the larger one is a DRAM access of its own it takes 8.1 times as long."""
    ms = [lib.time_resident(query.star(n, 1), capi.GPUQO_DPSUB, bicc=True, warmup=2, iters=5)[1] for n in (24, 26)]
    assert ms[1] < 6.0 * ms[0]
