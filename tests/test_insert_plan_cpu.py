"""When a bulk insert is a heap build (gpuheap_gb300/csrc/insert_plan.h),
compiled here by the host compiler: at the edges of the rule, for any sizes
without overflow, and the batches beside them inserted one by one."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include "insert_plan.h"
int main() {
    long long t, b, m, n;
    while (std::scanf("%lld %lld %lld %lld", &t, &b, &m, &n) == 4)
        std::printf("%d\n", gh::impl::build_pays(t != 0, b, m, n));
}
"""


@pytest.fixture(scope="module")
def pays(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("plan")
    src, exe = d / "plan.cpp", d / "plan"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "gpuheap_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)

    def ask(cases):
        text = "".join(" ".join(map(str, c)) + "\n" for c in cases)
        return [int(x) for x in subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True).stdout.split()]
    return ask


def test_a_few_batches_into_a_small_heap_go_one_by_one(pays):
    """One to four batches into 20 nodes and more took up to twice as long as
    a build, whatever the node size and layout."""
    few = [(t, b, m, n) for t in (0, 1) for b in (64, 1024, 16384) for m in (1, 2, 3, 4) for n in (20, 40, 100, 1000)]
    assert pays(few) == [0] * len(few)


@pytest.mark.parametrize("top,node,m,most", [(0, 2048, 4, 4), (0, 2048, 8, 32), (0, 2048, 16, 256), (0, 8192, 63, 47 * 63),
                                             (0, 64, 8, 16), (0, 64, 64, 5 * 64), (0, 64, 512, 23 * 512), (0, 512, 64, 23 * 64),
                                             (0, 8192, 1 << 20, 47 << 20), (1, 64, 4, 16), (1, 64, 16, 47 * 16), (1, 64, 64, 47 * 64)])
def test_edges(pays, top, node, m, most):
    assert pays([(top, node, m, most), (top, node, m, most + 1), (top, node, m, 0)]) == [1, 0, 1]


def test_no_overflow_at_the_largest_sizes(pays):
    big = (2**31) // 2 - 3
    assert pays([(0, 32768, big, 0), (0, 64, big, 1), (1, 64, 1, big), (0, 64, 2, big), (0, 64, 3, big)]) == [1, 1, 0, 0, 0]
