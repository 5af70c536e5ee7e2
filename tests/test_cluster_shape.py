"""The number of blocks of a BFS cluster: what the graph's size and the number
of sources ask for, as far as the device can run it; where it can run none, the
graph goes to the grid forms.  The rule is compiled for the host and the device
is a limit on the size."""
import itertools
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "cluster_shape.hpp"
int main(int argc, char** argv) {
    for (int i = 1; i + 2 < argc; i += 3) {
        const uint64_t n = std::strtoull(argv[i], nullptr, 10);
        const uint32_t k = std::atoi(argv[i + 1]), most = std::atoi(argv[i + 2]);
        std::printf("%u\n", gb::clusterSize(n, k, 148, [&](uint32_t nc) { return nc <= most; }));
    }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "shape.cpp").write_text(SRC)
    exe = str(d / "shape")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "graph_analytics_applesilicon_b200", "csrc"),
                    str(d / "shape.cpp"), "-o", exe], check=True)

    def ask(cases):
        args = [str(x) for c in cases for x in c]
        return [int(x) for x in subprocess.run([exe] + args, check=True, capture_output=True, text=True).stdout.split()]
    return ask


ROOM = (220 * 1024 - 32 * 2048) * 8  # vertices whose bitmap one block holds


def test_sizes(rule):
    ns = [1, 32767, 32768, 65536, 262143, 262144, ROOM, ROOM + 1, 2 * ROOM, 2 * ROOM + 33, 16 * ROOM, 16 * ROOM + 513]
    cases = list(itertools.product(ns, [1, 5, 20, 64], [16, 8, 4, 2, 1, 0]))
    for (n, k, most), got in zip(cases, rule(cases)):
        least = next((b for b in (1, 2, 4, 8, 16) if (n + 31) // 32 <= b * (ROOM // 32)), None)
        want = max([b for b in (1, 2, 4, 8, 16) if b == 1 or (k * b <= 148 and n >= b * 16384)])
        if least is None or most < least:
            assert got == 0, (n, k, most, got)
        else:
            assert got == min(max(want, least), most), (n, k, most, got)
