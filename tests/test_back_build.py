"""The stage-1 back kernel's build is chosen launch by launch (back_pixel_pairs of csrc/kernels.h, compiled here for the
host): two pixel pairs a thread where every SM has two tiles of that launch, one below and with the learned gate."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "compactcnncascade_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "kernels.h"
int main(int n, char** v) {
    for (int i = 2; i < n; ++i) std::printf("%d %d ", ccnn::back_pixel_pairs(atoi(v[i]), atoi(v[1]), false), ccnn::back_pixel_pairs(atoi(v[i]), atoi(v[1]), true));
    return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")), reason="no CUDA headers")
def test_rule(tmp_path):
    src, exe = tmp_path / "b.cpp", tmp_path / "b"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, "-I", os.path.join(CUDA, "include"), "-o", str(exe), str(src)])

    def pairs(sms, *tiles):
        v = list(map(int, subprocess.check_output([str(exe), str(sms)] + [str(t) for t in tiles]).split()))
        assert v[1::2] == [1] * len(tiles)
        return v[0::2]

    # the three launches of a 3840x2160 frame's 83 levels, and the edge
    assert pairs(148, 19263, 904, 44, 1, 295, 296) == [2, 2, 1, 1, 1, 2]
    assert pairs(132, 263, 264) == [1, 2]


def test_a_launch_s_own_tiles_decide():
    text = open(os.path.join(CSRC, "k_stage1.cu")).read()
    body = text[text.index("cudaError_t launch_stage1_back("):text.index("cudaError_t launch_stage1(")]
    assert "back_pixel_pairs(blocks, sms, back_on != nullptr)" in body[body.index("launch_grouped("):]
