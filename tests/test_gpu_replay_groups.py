"""The replay's routes through the list of boxes (up to 32, groups of up to and over 32, up to and over 512 boxes;
levels of a few and of many candidates; candidates tested against earlier boxes or not): the raw list and the
faces equal the oracle's."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import compactcnncascade_b200 as ccnn  # noqa: E402
from compactcnncascade_b200 import _capi  # noqa: E402
from oracle import oracle as orc  # noqa: E402


# few boxes; one face over 50 levels (its boxes are one group); some; hundreds; hundreds in small levels
@pytest.mark.parametrize("w,h,nf,lo,hi,min_face,scale", [(200, 160, 1, 60, 90, 30, 1.03), (400, 300, 2, 120, 200, 60, 1.02), (640, 480, 6, 40, 120, 30, 1.05),
                                                         (1280, 720, 60, 30, 90, 24, 1.05), (640, 480, 40, 24, 60, 20, 1.03)])
@pytest.mark.parametrize("drop,neighbors", [(1, 2), (0, 2), (1, 1), (0, 3)])
def test_lists(w, h, nf, lo, hi, min_face, scale, drop, neighbors):
    img, _ = ccnn.synth_frame(w, h, w + nf, nf, lo, hi)
    exp = orc.detect(img, min_face=min_face, max_face=240, scale_factor=scale, max_w=w, max_h=h, drop_detect=drop, min_neighbors=neighbors)
    p = ccnn.default_params()
    p.max_image_width, p.max_image_height = w, h
    p.min_face_height, p.max_face_height, p.scale_factor = min_face, 240, scale
    p.drop_detect, p.min_neighbors, p.detect_mode = drop, neighbors, 1
    det = ccnn.FaceDetector()
    assert det.Init(p) == 0, _capi.last_error()
    faces = det.Detect(img)
    assert det.raw_detections() == exp["raw"]
    assert [tuple(f) for f in faces] == exp["final"]
