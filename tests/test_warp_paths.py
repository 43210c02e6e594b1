"""Where a whole warp has to go one way: the listing loop of the sparse
memo's persistent kernel, which other blocks' counts can end in any iteration.
The sources are checked on the CPU (a warp that parts in front of a full-mask
exchange never returns, so it is not tried out); the kernel runs on a GPU at
every number of sets at which its arrays can run out."""
import os
import re

import pytest

from conftest import REPO, same_tree

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
