"""Boxes whose areas or common bounding boxes reach 2^24 pixels, where the drop test and the merges compare quotients
in floats instead of integers: the raw list and the faces of whole frames are the oracle's."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import compactcnncascade_b200 as ccnn  # noqa: E402
from compactcnncascade_b200 import _capi  # noqa: E402
from oracle import oracle as orc  # noqa: E402


# a frame is a small one with every pixel k x k times
@pytest.mark.parametrize("k,w,h,nf,lo,hi,min_face,scale,drop,seed", [(25, 400, 384, 2, 130, 220, 3600, 1.06, 1, 4), (25, 400, 384, 1, 180, 240, 4300, 1.05, 0, 3),
                                                                   (25, 400, 384, 1, 180, 240, 4300, 1.05, 1, 4)])
def test_large_boxes(k, w, h, nf, lo, hi, min_face, scale, drop, seed):
    small, _ = ccnn.synth_frame(w, h, seed, nf, lo, hi)
    img = np.ascontiguousarray(small.repeat(k, 0).repeat(k, 1))
    w, h = k * w, k * h
    exp = orc.detect(img, min_face=min_face, max_face=0, scale_factor=scale, max_w=w, max_h=h, drop_detect=drop)
    boxes = [(x, y, x + bw, y + bh) for x, y, bw, bh, *_ in exp["raw"]]
    # some overlapping pair's bounding box is past the integers' range
    assert any(min(a[2], b[2]) > max(a[0], b[0]) and min(a[3], b[3]) > max(a[1], b[1]) and
               (max(a[2], b[2]) - min(a[0], b[0])) * (max(a[3], b[3]) - min(a[1], b[1])) >= 1 << 24 for a, b in itertools.combinations(boxes, 2))
    p = ccnn.default_params()
    p.max_image_width, p.max_image_height = 640, 480  # the frame makes the detector grow, with one frame slot
    p.min_face_height, p.max_face_height, p.scale_factor = min_face, 0, scale
    p.drop_detect, p.detect_mode = drop, 1
    det = ccnn.FaceDetector()
    assert det.Init(p, schedule={"frame_slots": 1}) == 0, _capi.last_error()
    t = torch.from_numpy(img).cuda()
    faces = det.DetectDevice(t.data_ptr(), w, h, 3, 3 * w)
    assert det.raw_detections() == exp["raw"]
    assert faces == exp["final"] and faces
    det.Clear()
