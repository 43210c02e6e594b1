"""Where a whole warp has to go one way: the listing loop of the sparse
memo's persistent kernel, which other blocks' counts can end in any iteration,
and the hardware barrier of the queries that run as one cluster.  The sources
are checked on the CPU (a warp that parts in front of a full-mask exchange
never returns, so it is not tried out); on a GPU the listing kernel runs at
every number of sets at which its arrays can run out, and clusters of every
size against the oracle."""
import os
import re

import pytest

from conftest import REPO, same_tree

import harness
from gpuqo_b200 import capi, lib, query

CSRC = os.path.join(REPO, "postgres-gpuqo_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_listing_loop_leaves_as_a_warp():
    """The count that ends the loop is loaded by one lane and handed out."""
    source = _source("dp_wide.cu")
    kernel = source[source.index("k_wide_cactus(const"):source.index("#define CKW")]
    loop = kernel[kernel.index("nwarps - 1u - gwarp"):kernel.index("if (k >= 2u)")]
    loads = re.findall(r"([^;{}]*)__ldcg\(&ctl->level_n", loop)
    assert len(loads) == 1 and re.search(r"if \(lane == 0u\) listed = $", loads[0])
    assert re.search(r"if \([^;]*__shfl_sync\(kFullW, listed, 0\)[^;]*\) break;", loop)


def _level_counts(q):
    """connected sets of every size"""
    adj = [sum(1 << v for v in q.edges[u]) for u in range(q.n)]
    level, counts = {1 << v for v in range(q.n)}, [q.n]
    while len(counts) < q.n:
        level = {s | 1 << v for s in level for v in range(q.n) if not (s >> v) & 1 and adj[v] & s}
        counts.append(len(level))
    return counts


@pytest.mark.gpu
@pytest.mark.parametrize("shape,n", [("key_cycle", 37), ("ring_path", 33)])
def test_arrays_end_at_any_level(shape, n):
    q = query.make(shape, n, 5)
    want = lib.run(q, capi.GPUQO_DPSUB, bicc=True)
    assert want.error == 0 and want.stats["kernel_launches"] == 1
    counts, ends = _level_counts(q), []
    for c in counts:
        ends.append(c + (ends[-1] if ends else 0))
    L = lib.load()
    try:
        for room in sorted({e + d for e in ends for d in (-1, 0, 1)}):
            capi.set_int(L, "gpuqo_b200_sparse_host_list", room)
            got = lib.run(q, capi.GPUQO_DPSUB, bicc=True)
            assert got.error == 0 and same_tree(got.tree, want.tree)
            assert got.stats["connected_sets"] == sum(counts[1:])
            assert (got.stats["kernel_launches"] == 1) == (room >= ends[-1])
    finally:
        capi.set_int(L, "gpuqo_b200_sparse_host_list", 0)


def test_cluster_barrier_takes_a_warp_in_parts():
    """The barrier follows code that single lanes leave (a set's winner, a
    list's entries): .aligned would ask the warp to arrive as a whole."""
    source = _source("dp_barrier.cuh")
    assert len(re.findall(r"barrier\.cluster\.(?:arrive|wait)\.(?:release|acquire)", source)) == 2
    assert not re.search(r"barrier\.cluster[.\w]*\.aligned", source)


# queries small enough for one block or one cluster: a tree's level of up to
# 4096 splits, a cycle's every level
@pytest.mark.gpu
@pytest.mark.parametrize("shape,sizes", [("star", range(2, 13)), ("snowflake", (5, 9, 14, 17)),
                                         ("key_chain", (2, 7, 16, 30)), ("cycle", (3, 4, 9, 15)),
                                         ("key_cycle", (5, 12, 16))])
def test_clusters(shape, sizes):
    for n in sizes:
        for rich in (False, True):
            q = query.make(shape, n, 11, rich=rich)
            for alg in ((5, 3) if n <= 13 else (5,)):
                want = harness.run_port(q, alg)[0]
                for _ in range(3):
                    got = lib.run(q, capi.GPUQO_DPSUB, bicc=(alg == 5))
                    assert got.error == 0 and same_tree(got.tree, want)
