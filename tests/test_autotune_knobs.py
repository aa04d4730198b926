"""Every value the tuner tries for the persistent stage-1 kernel's grid is a grid of its own: twice the value in blocks
of 128 threads a SM, at most what the kernel's register bound lets reside."""
import os
import re

from compactcnncascade_b200 import autotune

CSRC = os.path.join(os.path.dirname(os.path.abspath(autotune.__file__)), "csrc")


def test_batch_blocks_values_are_distinct():
    text = open(os.path.join(CSRC, "k_stage1.cu")).read()
    fit = int(re.search(r"__launch_bounds__\(kBatchThreads, (\d+)\) stage1_batch_kernel", text).group(1))
    values = dict(autotune.KNOBS)["batch_blocks_per_sm"]
    assert len({min(2 * v, fit) for v in values}) == len(values)
    assert max(min(2 * v, fit) for v in values) == fit
