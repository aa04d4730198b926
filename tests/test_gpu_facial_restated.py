"""Facial analysis against the float32 restatement of its network (oracle/facial_ref.py) on the detector's own
candidates: which windows are dropped, the raw list, and every face's box, score and attributes."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import compactcnncascade_b200 as ccnn  # noqa: E402
from compactcnncascade_b200 import _capi  # noqa: E402
from oracle import facial_ref  # noqa: E402
from oracle import oracle as orc  # noqa: E402

F = np.float32
NET = facial_ref.load(os.path.join(os.path.dirname(os.path.abspath(ccnn.__file__)), "models", "cnn4landmarks_cntk.bin"))


def window(px, py, inv, retry, gw, gh, pattern=(23, 27)):
    """The check window of a candidate in the gray frame (cnn_detector_v3.cpp:1489-1556): x, y, cols, rows."""
    x, y, w, h = int(F(px - 6) * inv), int(F(py - 5) * inv), int(F(pattern[0] + 13) * inv), int(F(pattern[1] + 11) * inv)
    if retry:
        k = F(0.15)
        x, w = int(F(x) + F(w) * k / F(2)), int(F(w) - F(w) * k)
        y, h = int(F(y) + F(h) * k / F(2)), int(F(h) - F(h) * k)
    rx, ry = min(max(x, 0), gw), min(max(y, 0), gh)
    return rx, ry, min(max(x + w, 0), gw) - rx, min(max(y + h, 0), gh) - ry


# boxes of a frame: few, many, more than the 512 whose attributes are gathered into shared memory
@pytest.mark.parametrize("w,h,nf,lo,hi,min_face,scale,precision,at_least", [(640, 480, 5, 40, 200, 40, 1.15, 3, 4), (640, 480, 5, 40, 200, 40, 1.1, 2, 10),
                                                                          (1280, 720, 30, 40, 160, 40, 1.1, 4, 30), (400, 300, 20, 24, 60, 20, 1.007, 3, 513)])
def test_faces_and_attributes(w, h, nf, lo, hi, min_face, scale, precision, at_least):
    img, _ = ccnn.synth_frame(w, h, 77, nf, lo, hi)
    p = ccnn.default_params()
    p.max_image_width, p.max_image_height = w, h
    p.min_face_height, p.max_face_height, p.scale_factor = min_face, 240, scale
    p.detect_precision, p.detect_mode, p.facial_analysis = precision, 1, 1
    det = ccnn.FaceDetector()
    assert det.Init(p) == 0, _capi.last_error()
    got = det.Detect(img, attributes=True)
    scales = [F(lv[2]) for lv in det.levels()]
    gray = det.getGrayImage32F()
    raw, attributes = [], []
    for level, px, py, _, accepted, score, knn in det.candidates():
        if not accepted:
            continue
        inv = F(1) / scales[level]
        x, y, cols, rows = window(px, py, inv, accepted == 2, gray.shape[1], gray.shape[0])
        dropped, *values = facial_ref.analyse(NET, orc.resize_f32(gray[y:y + rows, x:x + cols], 49, 51, 0), cols, rows)
        if not dropped:
            raw.append((int(F(px) * inv), int(F(py) * inv), int(F(23) * inv), int(F(27) * inv), score, float(scales[level]), knn, 0))
            attributes.append(tuple(values))
    assert len(raw) >= at_least
    assert det.raw_detections() == raw
    order = [len(raw) - 1 - k for k in orc.sort_perm([r[5] for r in reversed(raw)])]
    boxes = [(r[0], r[1], r[0] + r[2], r[1] + r[3], r[4]) for r in (raw[k] for k in order)]
    if precision == 4:  # clusters of fewer than two merges leave between the merges
        keep = [own for own in facial_ref.merger(boxes, 0.5, False)[1] if len(own) > 2]
        clusters = {m for own in keep for m in own}
        order, boxes = [k for m, k in enumerate(order) if m in clusters], [b for m, b in enumerate(boxes) if m in clusters]
    assert got == facial_ref.faces(boxes, [attributes[k] for k in order]) and got
