"""Kernels that start while the one before them ends (they call chain_wait) read what earlier kernels wrote by
ordinary loads only: __ldg and const __restrict__ pointers ask that the data stay the same for as long as the kernel
is resident, and a wait does not order them. Read from the sources: every such kernel and the device functions it
calls."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "compactcnncascade_b200", "csrc")
HEADERS = ("ccnn_common.cuh", "legacy_dev.cuh", "resample.cuh", "replay.cuh", "window_common.cuh", "pyramid.cuh")
# written when a plan or a detector is made, before any launch that reads them: scan chunks, level descriptors, networks
CONSTANT = {"chunks", "levels", "N", "Np", "G"}


def _functions(name):
    """(name, whole text) of the file's __global__ and __device__ functions."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*|__launch_bounds__\([^)]*\)", "", f.read())
    out = []
    for m in re.finditer(r"__(?:global|device)__[^;{}()]*?\b(\w+)\(", text):
        depth, i = 1, m.end()
        while depth:  # to the end of the parameters
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        j = i + re.match(r"\s*", text[i:]).end()
        if text[j] != "{":
            continue
        depth, k = 1, j + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        out.append((m.group(1), text[m.start():k]))
    return out


def _chained(name):
    """The texts of the file's chained kernels and of what they call, by function name."""
    every = [f for h in HEADERS for f in _functions(h)] + _functions(name)
    todo = [(n, t) for n, t in _functions(name) if "chain_wait();" in t]
    kernels = [n for n, _ in todo]
    seen = {}
    while todo:
        n, t = todo.pop()
        if (n, t) in seen:
            continue
        seen[(n, t)] = True
        todo += [(m, u) for m, u in every if m != n and re.search(r"\b%s\b\s*(?:<[^;(]*>)?\(" % m, t)]
    return kernels, list(seen)


@pytest.mark.parametrize("name,kernels", [("k_stage1.cu", {"stage1_front_kernel", "stage1_back_kernel"}), ("k_candidates.cu", {"cand_write_kernel"}),
                                          ("k_window.cu", {"window_kernel"}), ("k_facial.cu", {"facial_kernel"}), ("k_replay.cu", {"replay_kernel"}),
                                          ("gate.cu", {"gate_mask_kernel"}), ("k_legacy.cu", {"legacy_pool_kernel", "legacy_out_kernel"})])
def test_ordinary_loads(name, kernels):
    found, functions = _chained(name)
    assert set(found) == kernels
    bad = []
    for fn, text in functions:
        bad += [(fn, p) for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", text) if p not in CONSTANT]
        # fields of a network only
        bad += [(fn, a) for a in re.findall(r"__ldg\(([^\n]{0,30})", text) if not re.match(r"&(?:W|N|G)(?:\.|->)", a)]
    assert not bad


def test_no_other_file_launches_chained_kernels():
    users = {f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and "launch_chained(" in open(os.path.join(CSRC, f)).read()}
    assert users == {"k_stage1.cu", "k_candidates.cu", "k_window.cu", "k_facial.cu", "k_replay.cu", "gate.cu", "k_legacy.cu"}
