"""The host's choice of how a bulk delete runs (gpuheap_gb300/csrc/
delete_plan.h), compiled here by the host compiler and asked at the edges of
its rules."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "delete_plan.h"
using namespace gh::impl;
int main(int argc, char** argv) {
    long long a[8] = {};
    for (int i = 1; i < argc && i <= 8; ++i) a[i - 1] = std::atoll(argv[i]);
    std::printf("%d\n", drains_whole(a[0], a[1], static_cast<int>(a[2])));
    if (argc > 4) std::printf("%lld\n", out_piece(a[0], a[3], static_cast<int>(a[4]), false));
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("plan")
    src, exe = d / "plan.cpp", d / "plan"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "gpuheap_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    return lambda *a: [int(x) for x in subprocess.run([str(exe)] + [str(x) for x in a], check=True, capture_output=True,
                                                      text=True).stdout.split()]


@pytest.mark.parametrize("keys,whole", [(3 * 2048, 0), (4 * 2048, 1), (2**31 - 1, 1), (2**31, 0), (2**32, 0), (2**32 + 2**20, 0),
                                        (3 * 2**31, 0)])
def test_one_sort_empties_heaps_of_4_nodes_to_2e31_keys(plan, keys, whole):
    """An output limit is an int: a sort of 2^31 keys and more would not start,
    and gh_heap_sort_host would copy out what its buffer held before."""
    assert plan(keys, keys // 2048, 4) == [whole]


@pytest.mark.parametrize("keys,B", [(2**31 - 1, 2048), (2**31, 16), (2**34 + 5, 4096), (2**34 + 2**33, 2048), (2**35, 256)])
def test_pieces_of_whole_batches_that_an_int_counts(plan, keys, B):
    piece = -(-(-(-keys // 8)) // B) * B  # an eighth, in whole batches
    got = plan(keys, keys // B, 4, piece, B)[1]
    assert got % B == 0 and 0 < got <= 2**31 - 1 and got <= piece
    assert got == piece or got + B > 2**31 - 1
