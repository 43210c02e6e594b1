"""CPU: an allocation that fails leaves the engines usable.  Every allocation
of a call fails in turn, under a stand-in for the CUDA runtime that does
nothing but hold memory and watch the pointers it is given (fake_cudart.cpp); a
smaller call after it must neither free a buffer again nor launch on one that
is not there."""
import json
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

import pytest

from conftest import REPO

ERR_NOMEM = 3

CHILD = """
import ctypes, json, sys
from gpuqo_b200 import capi, lib, query
kind, fail = sys.argv[1], int(sys.argv[2])
fake = ctypes.CDLL(sys.argv[3])
var = lambda name: ctypes.c_int.in_dll(fake, name)
def call(size):
    if kind == "tree":
        return lib.run(query.snowflake(size, 1), capi.GPUQO_DPSUB, bicc=True).error
    if kind == "dpsize":
        return lib.run(query.clique(size, 1), capi.GPUQO_DPSIZE).error
    queries = {"trees": [query.star(size, 1), query.snowflake(size - 1, 2)],
               "cliques": [query.clique(size, 1), query.cycle(size - 1, 2)]}[kind]
    return lib.run_batch(queries, capi.GPUQO_DPSUB, bicc=True)[1]
var("fake_fail_from").value, var("fake_fail_count").value = fail, 2   # and the next: a smaller try at the same buffer
before = [call(8), call(17)]
total = var("fake_allocations").value
var("fake_fail_from").value = -1
after = [call(n) for n in (8, 14, 18)]
print(json.dumps([total, before, after, var("fake_bad").value, var("fake_launches").value]))
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", out, os.path.join(REPO, "tests", "fake_cudart.cpp")],
                   check=True)
    return out


def _child(fake, kind, fail):
    env = dict(os.environ, LD_PRELOAD=fake, PYTHONPATH=os.path.join(REPO, "postgres-gpuqo_b200"))
    done = subprocess.run([sys.executable, "-c", CHILD, kind, str(fail), fake], env=env, capture_output=True, text=True,
                          timeout=120)
    assert done.returncode == 0, done.stderr
    return json.loads(done.stdout)


@pytest.mark.parametrize("kind", ["tree", "trees", "cliques", "dpsize"])
def test_smaller_calls_after_a_failed_allocation(fake, kind):
    total, before, after, bad, launches = _child(fake, kind, -1)
    assert bad == 0 and launches > 0 and total > 0 and ERR_NOMEM not in before + after
    with ThreadPoolExecutor(8) as pool:
        runs = list(pool.map(lambda fail: _child(fake, kind, fail), range(total)))
    for fail, (_, failed, then, bad, _) in enumerate(runs):
        assert ERR_NOMEM in failed and all(f in (b, ERR_NOMEM) for f, b in zip(failed, before)), fail
        assert then == after and bad == 0, fail


REFUSED = """
import sys
from gpuqo_b200 import capi, lib, query
big = query.star(12, 1)
first = list(big.eq_classes)
for i in range(6000):   # a planner info larger than a block's shared memory
    big.eq_classes.append(query.EqClass(list(first[i % 11].members), [0.5], [[], []], [query.VarInfo()] * 2))
for q in (query.star(12, 1), big, query.star(12, 1)):
    print("call", lib.run(q, capi.GPUQO_DPSUB, bicc=True).error, file=sys.stderr)
"""


def test_a_refused_call_leaves_no_error_for_the_next(fake):
    env = dict(os.environ, LD_PRELOAD=fake, PYTHONPATH=os.path.join(REPO, "postgres-gpuqo_b200"))
    done = subprocess.run([sys.executable, "-c", REFUSED], env=env, capture_output=True, text=True, timeout=120)
    _, refused, after = done.stderr.split("call 2\n")[:3]
    assert done.returncode == 0 and "cudaFuncSetAttribute" in refused
    # no plan comes from kernels that do nothing, but the runtime has no complaint
    assert "nodes" in after and "cuda" not in after


MANY_CLASSES = """
import ctypes, json, sys
from gpuqo_b200 import capi, lib, query
fake = ctypes.CDLL(sys.argv[1])
launches = ctypes.c_int.in_dll(fake, "fake_launches")
def call(n, classes, persistent, extra=()):   # 1,100 classes: a planner info of some 90 KB
    L = lib.load()
    L.gpuqo_b200_reset_persistent()   # no plan comes from the kernels here, which counts as a barrier that gave up
    capi.set_int(L, "gpuqo_b200_persistent", persistent)
    q = query.star(n, 1)
    for a, b in extra:
        q.edges[a], q.edges[b] = sorted(q.edges[a] + [b]), sorted(q.edges[b] + [a])
    first = list(q.eq_classes)
    for i in range(classes - len(first)):
        q.eq_classes.append(query.EqClass(list(first[i % len(first)].members), [0.5], [[], []], [query.VarInfo()] * 2))
    before = launches.value
    lib.run(q, capi.GPUQO_DPSUB, bicc=True)
    return launches.value - before
"""


def _many_classes(fake, calls):
    env = dict(os.environ, LD_PRELOAD=fake, PYTHONPATH=os.path.join(REPO, "postgres-gpuqo_b200"))
    done = subprocess.run([sys.executable, "-c", MANY_CLASSES + f"print(json.dumps({calls}))", fake], env=env,
                          capture_output=True, text=True, timeout=120)
    assert done.returncode == 0
    return json.loads(done.stdout), done.stderr


def test_a_smaller_planner_info_leaves_the_larger_one_its_shared_memory(fake):
    """the level kernels that follow are in a captured graph by the third call: its one launch is the persistent
    kernel's, with the shared memory that the second call's size would not allow"""
    launched, _ = _many_classes(fake, "[call(12, 1100, 1), call(12, 850, 1), call(12, 1100, 1)]")
    assert launched[2] == 1


def test_level_kernels_are_allowed_the_planner_info(fake):
    """a tree, and a graph with a cycle, by the launches per level"""
    launched, said = _many_classes(fake, "[call(12, 1100, 0), call(12, 1100, 0, [(0, 1), (0, 2), (1, 2)])]")
    assert min(launched) > 0 and "cuda" not in said
