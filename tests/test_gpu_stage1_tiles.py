"""Stage-1 response maps where the tiles of the front (32 x 16 pooled pixels) and back (32 x 16 responses)
kernels end: maps of one row or column, of one more or less than a tile or half a tile, and frames on both
sides of the back kernel's choice between one and two pixel pairs a thread. Every map equals the oracle's
bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import compactcnncascade_b200 as ccnn  # noqa: E402
from compactcnncascade_b200 import _capi  # noqa: E402
from oracle import oracle as orc  # noqa: E402


def _image_side(responses, extra, halo):
    """The image side whose map has that many responses (extra: 0-3 leftover pixels)."""
    return ((responses + halo) * 2 + 2) * 2 + 3 + extra


@pytest.mark.parametrize("ow,oh,extra,pad", [(1, 1, 0, 0), (15, 3, 1, 1), (16, 16, 2, 0), (17, 17, 3, 4), (31, 5, 0, 3), (33, 15, 1, 0), (64, 33, 0, 0),
                                             (47, 20, 3, 0), (200, 130, 1, 0), (640, 300, 0, 0), (641, 301, 3, 2)])
def test_stored_image(ow, oh, extra, pad):
    w, h = _image_side(ow, extra, 3), _image_side(oh, (extra * 3) % 4, 4)
    rng = np.random.default_rng(100 * ow + oh)
    img = (rng.random((h, w), dtype=np.float32) * 255).astype(np.float32)
    exp = orc.net_forward(1, img, 1)
    assert exp.shape == (oh, ow)
    buf = torch.zeros((h, w + pad), dtype=torch.float32, device="cuda")
    buf[:, :w] = torch.from_numpy(img)
    out = torch.zeros(ow * oh, dtype=torch.float32, device="cuda")
    det = ccnn.FaceDetector()
    assert det.Init(ccnn.default_params()) == 0, _capi.last_error()
    rw, rh = ctypes.c_int(), ctypes.c_int()
    st = _capi.lib().ccnn_stage1_forward(det._h, buf.data_ptr(), w, h, (w + pad) * 4, out.data_ptr(), ow * oh, ctypes.byref(rw), ctypes.byref(rh), None)
    assert st == 0, _capi.last_error()
    assert (rw.value, rh.value) == (ow, oh)
    assert np.array_equal(out.cpu().numpy().reshape(oh, ow).view(np.uint32), exp.view(np.uint32))


# copy, nearest-neighbour and bilinear levels, ragged tiles; the last has more than 296 back tiles
@pytest.mark.parametrize("w,h,channels,min_face,scale", [(47, 51, 1, 27, 1.15), (150, 83, 3, 27, 1.3), (211, 331, 3, 24, 1.1), (333, 222, 4, 40, 1.2),
                                                         (1333, 1001, 3, 27, 1.05)])
@pytest.mark.parametrize("batch_frames", [0, 1])
def test_frame(w, h, channels, min_face, scale, batch_frames):
    img, _ = ccnn.synth_frame(w, h, 3 * w + h, 4, 30, max(34, min(w, h) // 2), channels=channels)
    exp = orc.detect(img, min_face=min_face, max_face=240, scale_factor=scale, max_w=w, max_h=h)
    p = ccnn.default_params()
    p.max_image_width, p.max_image_height = w, h
    p.min_face_height, p.max_face_height, p.scale_factor = min_face, 240, scale
    det = ccnn.FaceDetector()
    assert det.Init(p, schedule={"frame_slots": 2, "batch_frames": batch_frames}) == 0, _capi.last_error()
    faces = det.Detect(img)
    assert len(det.levels()) == len(exp["levels"]) > 0
    for i, r in enumerate(exp["resp"]):
        assert np.array_equal(det.response_map(i).view(np.uint32), r.view(np.uint32)), (i, exp["levels"][i])
    assert [tuple(f) for f in faces] == exp["final"]
