"""GPU: row widths around the places where a row's byte size changes its form
(below zero, where the reference's 64-bit sum wraps or stays near 2^64, and
around the alignment), on every kernel that costs pages, against the oracle.
work_mem is small, so that hash joins take several batches and read pages."""
import ctypes as C

import pytest

from conftest import same_tree

import harness
from gpuqo_b200 import capi, lib, query

pytestmark = pytest.mark.gpu

QUERIES = {"tree": (lambda: query.snowflake(10, 3), (5, 3)), "tree_stats": (lambda: query.star(9, 4, rich=True), (5, 3)),
           "cycle": (lambda: query.key_cycle(9, 5), (5, 3)), "random": (lambda: query.random_graph(9, 6, 0.3, rich=True), (5, 3)),
           "clique": (lambda: query.clique(7, 7), (5, 3))}


@pytest.fixture
def small_work_mem():
    saved = [(v, v.value) for v in (C.c_int.in_dll(library, "work_mem") for library in (lib.load(), harness.load_port()))]
    for var, _ in saved:
        var.value = 64
    yield
    for var, value in saved:
        var.value = value


@pytest.mark.parametrize("width", [-2147483648, -2147483640, -100000, -33, -32, -31, -25, -24, -23, -9, -8, -7, -1, 0, 1, 7, 8, 9])
@pytest.mark.parametrize("name", sorted(QUERIES))
def test_width(name, width, small_work_mem):
    make, algs = QUERIES[name]
    q = make()
    q.width = [width if i % 3 else 8 for i in range(q.n)]
    if width < -2147480000:   # one such row: the widths of a set are summed in 32 bits
        q.width = [8] * (q.n - 1) + [width]
    for alg in algs:
        want = harness.run_port(q, alg)[0]
        got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
        assert got.error == 0 and same_tree(got.tree, want)
