"""Heap::exchangeMin (insert and take in one pass through the heap's top) and
the inserts that leave the partial buffer alone, driven from a user program's
own kernels (tests/compat/exchange.cu) against a host multiset: both layouts,
batch sizes 64 to 2048, one block and several, with and without a threshold,
few distinct keys and many."""
import os
import subprocess

import pytest

from test_compat_adapter import ARCH, REPO, _nvcc

SRC = os.path.join(REPO, "tests", "compat", "exchange.cu")
FLAGS = ["-std=c++17", "-O2", "-I" + os.path.join(REPO, "include")]


def test_exchange_program_compiles(tmp_path):
    r = subprocess.run([_nvcc()] + ARCH + FLAGS + ["-c", SRC, "-o", str(tmp_path / "x.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.gpu
def test_exchange_program_runs(tmp_path, ghlib):
    libdir = os.path.join(REPO, "gpuheap_gb300")
    exe = str(tmp_path / "exchange")
    r = subprocess.run([_nvcc()] + ARCH + FLAGS + [SRC, "-o", exe, "-L" + libdir, "-lgpuheap_gb300", "-Xlinker",
                                                   "-rpath=" + libdir], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "exchange ok" in run.stdout, run.stdout + run.stderr
