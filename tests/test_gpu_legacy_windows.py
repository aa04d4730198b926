"""The legacy (format 1.0) cascade inside the detector against the float32 restatement of its networks: every level's
response map and, candidate by candidate, the verdict of the stage-2/3 windows (accepted crop, score, count)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import compactcnncascade_b200 as ccnn  # noqa: E402
from compactcnncascade_b200 import _capi  # noqa: E402
from oracle import legacy_ref  # noqa: E402
from oracle import oracle as orc  # noqa: E402
from tests.test_gpu_facial_restated import window  # noqa: E402

F = np.float32
MODELS = [os.path.join(os.path.dirname(os.path.abspath(ccnn.__file__)), "models", f"cnn4face{i}_new.bin") for i in (1, 2, 3)]
NETS = [legacy_ref.load(m) for m in MODELS]


def _check(gray, cand, inv, retry, p):
    """(accepted, score, count) of one window with type_check 2 (cnn_detector_v3.cpp:1565-1725)."""
    _, px, py, score0 = cand[:4]
    x, y, cols, rows = window(px, py, inv, retry, gray.shape[1], gray.shape[0], NETS[0]["min"])
    u8 = (orc.resize_f32(gray[y:y + rows, x:x + cols], 49, 51, 0) + F(0.5)).astype(np.int32).astype(np.uint8)
    if p.equalize:
        assert orc.load().orc_equalize(u8.ctypes.data, 49, 51) == 0
    best, count = [F(-10), F(-10)], [0, 0]
    for stage, view in enumerate((u8[:, 2:], u8[:, 46::-1] if p.reflection else u8[:, :47])):
        out = legacy_ref.forward(NETS[1 + stage], view.astype(F))
        assert out.shape == (4, 4)
        best[stage], count[stage] = max(F(-10), out.max()), int((out > F(p.treshold[1 + stage])).sum())
        if count[stage] < max(1, p.min_neighbors):
            break
    score = (F(score0) + F(count[0]) * max(F(-1.7159), best[0])) + F(count[1]) * max(F(-1.7159), best[1])
    return min(count) >= p.min_neighbors, float(score), min(count)


@pytest.mark.parametrize("w,h,seed,nf,equalize,reflection,neighbors", [(320, 240, 1, 3, 1, 1, 2), (333, 211, 2, 3, 0, 1, 2), (320, 240, 3, 4, 1, 0, 1), (400, 301, 4, 4, 1, 1, 3)])
def test_cascade(w, h, seed, nf, equalize, reflection, neighbors):
    img, _ = ccnn.synth_frame(w, h, seed, nf, 40, 120)
    p = ccnn.default_params()
    p.max_image_width, p.max_image_height = w, h
    p.min_face_height, p.max_face_height, p.scale_factor, p.detect_mode = 40, 200, 1.15, 1
    p.equalize, p.reflection, p.min_neighbors = equalize, reflection, neighbors
    p.treshold[0] = -1.6
    det = ccnn.FaceDetector()
    assert det.Init(p, models=MODELS) == 0, _capi.last_error()
    det.Detect(img)
    gray, levels = det.getGrayImage32F(), det.levels()
    for i, (lw, lh, scale, rw, rh) in enumerate(levels):
        want = legacy_ref.forward(NETS[0], orc.resize_f32(gray, lw, lh, 0 if scale > F(0.7) else 1))
        got = det.response_map(i)
        assert got.shape == want.shape == (rh, rw) and np.array_equal(got.view(np.uint32), want.view(np.uint32)), i
    cands, yes = det.candidates(), 0
    assert cands
    for c in cands:
        inv = F(1) / F(levels[c[0]][2])
        for mod in (0, 1):
            ok, score, count = _check(gray, c, inv, mod == 1, p)
            if ok:
                break
        assert c[4] == (mod + 1 if ok else 0)
        if ok:
            yes += 1
            assert (c[5], c[6]) == (score, count)
    assert yes
