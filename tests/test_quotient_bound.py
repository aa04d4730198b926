"""The replay's division-free comparison (quot_gt_int of csrc/replay.cuh, compiled here for the host) equals the
float quotient's: at the thresholds of the cascade, for the integers on both sides of every boundary, for random
ones, and at the ends of the range."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "compactcnncascade_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <random>
#include "replay.cuh"
using namespace ccnn;
static long bad = 0, n = 0;
static void check(long a, long b, float t) {
    if (a < 0 || b <= 0 || a >= kQuotMax || b >= kQuotMax) return;
    uint32_t u;
    std::memcpy(&u, &t, 4);
    volatile float q = (float)a / (float)b;
    ++n;
    if (quot_gt_int((int)a, (int)b, quot_bound(u)) != (q > t)) ++bad;
}
int main() {
    std::mt19937 g(7);
    const float half = 0.5f, fifth = 0.2f, k = 0.75f;
    const float ts[] = {half, k * half, 0.7f, fifth, k * fifth, 1.f, 0x1p-12f, 0.99999994f};
    for (float t : ts) {
        for (long b = 1; b < kQuotMax; b += b < 5000 ? 1 : 1 + (long)(g() % 4001)) {
            const long a0 = (long)((double)t * (double)b);
            for (long d = -3; d <= 3; ++d) check(a0 + d, b, t);
            check(b, b, t);
            check(0, b, t);
            check((long)(g() % kQuotMax), b, t);
        }
        for (long d = 0; d < 2000; ++d) check((long)((double)t * (kQuotMax - 1)) - 1000 + d, kQuotMax - 1, t);
    }
    std::printf("%ld %ld\n", n, bad);
    return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")), reason="no CUDA headers")
def test_equals_the_float_quotient(tmp_path):
    src = tmp_path / "q.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "q"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, "-I", os.path.join(CUDA, "include"), "-o", str(exe), str(src)])
    n, bad = map(int, subprocess.check_output([str(exe)]).split())
    assert n > 400000 and bad == 0
