"""CPU: the host files are compiled for the machine that builds them, AVX2 where
it has it, and for any x86-64 host on request."""
import os
import subprocess

import pytest

from conftest import REPO

PKG = os.path.join(REPO, "postgres-gpuqo_b200")


@pytest.mark.parametrize("flags,settings,v3", [("fpu sse2 avx avx2 bmi2", [], True), ("fpu sse2 avx", [], False),
                                               ("fpu sse2 avx avx2 bmi2", ["HOST_ARCH="], False)])
def test_host_flags(flags, settings, v3, tmp_path):
    cpuinfo = tmp_path / "cpuinfo"
    cpuinfo.write_text("processor : 0\nflags\t\t: " + flags + "\n")
    lines = subprocess.run(["make", "-n", "-B", "-C", PKG, f"CPUINFO={cpuinfo}"] + settings, check=True,
                           capture_output=True, text=True).stdout.splitlines()
    for name in ("host_api", "host_idp", "host_serve"):
        assert ["x86-64-v3" in l for l in lines if f"/{name}.cpp -o" in l] == [v3]
    check = [l for l in lines if "/host_cpu.cpp -o" in l]
    assert len(check) == 1 and "-march" not in check[0] and ("GPUQO_HOST_X86_64_V3" in check[0]) == v3


def test_the_library_loads_without_a_word():
    """on this machine, which built it"""
    import sys
    done = subprocess.run([sys.executable, "-c", "from gpuqo_b200 import lib; lib.load()"], capture_output=True, text=True,
                          env=dict(os.environ, PYTHONPATH=PKG))
    assert done.returncode == 0 and "gpuqo_b200:" not in done.stderr
