"""The shares that blocks add to a completion counter (block_share in pps_internal.h), run on
the host: a launch elects its last block and no other, and launches that overlapped on one
counter leave it at zero, so that the next one elects right again."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include "pps_internal.h"
#include <cstdio>
#include <random>
#include <utility>
#include <vector>
using pps::block_share;

static unsigned counter = 0;
static bool count(unsigned bid, unsigned n)   // count_block, one caller at a time
{
    counter += block_share(bid, n);
    return counter == 0u;
}

int main()
{
    std::mt19937 rng(1);
    const unsigned sizes[] = {1, 2, 3, 31, 256, 1216, 16384};
    auto serial = [&](unsigned n) {   // blocks in any order: the last to count, and only it, is elected
        std::vector<unsigned> order(n);
        for (unsigned b = 0; b < n; b++) order[b] = b;
        for (unsigned b = n; b > 1; b--) std::swap(order[b - 1], order[rng() % b]);
        for (unsigned b = 0; b < n; b++)
            if (count(order[b], n) != (b == n - 1)) return false;
        return counter == 0u;
    };
    for (int round = 0; round < 20; round++)
        for (unsigned a : sizes)
            for (unsigned c : sizes) {
                if (!serial(a)) return 1;
                unsigned done[2] = {0, 0}, n[2] = {a, c};   // two launches that overlap
                while (done[0] < n[0] || done[1] < n[1]) {
                    int who = (int)(rng() % 2);
                    if (done[who] == n[who]) who = 1 - who;
                    count(done[who]++, n[who]);
                }
                if (counter != 0u || !serial(c)) return 2;
            }
    std::puts("ok");
    return 0;
}
"""


def test_counter_is_back_at_zero_after_any_launches(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not shutil.which("g++") or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "count.cpp", tmp_path / "count"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "parallelpoissonsolver_gb300", "csrc"), "-I",
                    os.path.join(cuda, "include"), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "ok\n"
