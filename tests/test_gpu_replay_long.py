"""The replay's routes for long lists against the oracle: levels of more than 256 candidates (one warp tests the
boxes), more than 128 levels (their scales are read from global memory), lists that do not fit in shared memory and
more than 512 boxes. The raw list and the faces are the oracle's."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import compactcnncascade_b200 as ccnn  # noqa: E402
from compactcnncascade_b200 import _capi  # noqa: E402
from oracle import oracle as orc  # noqa: E402

FITS = 1692  # candidates whose working set the replay keeps in shared memory


# the last four: whether the lists fit, the least candidates of the fullest level, levels and raw boxes of the route
@pytest.mark.parametrize("w,h,nf,lo,hi,min_face,scale,thr1,drop,fits,in_level,levels,raw", [
    (640, 480, 80, 30, 60, 40, 1.15, -1.7, 1, True, 257, 1, 1), (640, 480, 80, 30, 60, 40, 1.15, -1.7, 0, True, 257, 1, 1),
    (800, 600, 120, 30, 60, 40, 1.15, -1.7, 1, False, 257, 1, 1), (240, 200, 2, 40, 90, 20, 1.012, -1.5, 1, True, 1, 129, 1),
    (400, 300, 20, 24, 60, 20, 1.01, -1.5, 1, False, 1, 129, 513), (400, 300, 20, 24, 60, 20, 1.01, -1.5, 0, False, 1, 129, 1)])
def test_long_lists(w, h, nf, lo, hi, min_face, scale, thr1, drop, fits, in_level, levels, raw):
    img, _ = ccnn.synth_frame(w, h, 77, nf, lo, hi)
    exp = orc.detect(img, min_face=min_face, max_face=240, scale_factor=scale, max_w=w, max_h=h, drop_detect=drop, thr=(thr1, -1.25, -1.0), resp_cap=20 * w * h)
    per_level = {}
    for c in exp["candidates"]:
        per_level[c[0]] = per_level.get(c[0], 0) + 1
    # the frame takes the route
    assert (len(exp["candidates"]) <= FITS) == fits and max(per_level.values()) >= in_level
    assert len(exp["levels"]) >= levels and len(exp["raw"]) >= raw
    p = ccnn.default_params()
    p.max_image_width, p.max_image_height = w, h
    p.min_face_height, p.max_face_height, p.scale_factor = min_face, 240, scale
    p.drop_detect, p.detect_mode = drop, 1
    p.treshold[0] = thr1
    det = ccnn.FaceDetector()
    assert det.Init(p) == 0, _capi.last_error()
    faces = det.Detect(img)
    assert [c[:4] for c in det.candidates()] == exp["candidates"]
    assert det.raw_detections() == exp["raw"]
    assert [tuple(f) for f in faces] == exp["final"]
