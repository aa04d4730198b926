"""A frame of more than 2^32 pixels: level rows past that offset are sampled from the rows they belong to (faces are
only in the frame's last rows, the rest is black)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import compactcnncascade_b200 as ccnn  # noqa: E402
from compactcnncascade_b200 import _capi  # noqa: E402


def test_last_rows():
    w, h, pw, ph, x0 = 70016, 61760, 2400, 320, 30000
    y0 = h - ph
    assert w * y0 > 1 << 32
    if torch.cuda.mem_get_info()[0] < 125 << 30:
        pytest.skip("the frame and its detector need 100 GB of free device memory")
    frame = torch.zeros((h, w, 3), dtype=torch.uint8, device="cuda")
    patch, _ = ccnn.synth_frame(pw, ph, 9, 60, 42, 50)
    frame[y0:, x0:x0 + pw] = torch.from_numpy(patch).cuda()
    p = ccnn.default_params()
    p.max_image_width, p.max_image_height = 640, 480  # the frame makes the detector grow, with one frame slot
    p.min_face_height, p.max_face_height, p.scale_factor, p.detect_mode = 40, 41, 1.15, 1
    det = ccnn.FaceDetector()
    assert det.Init(p, schedule={"frame_slots": 1}) == 0, _capi.last_error()
    faces = det.DetectDevice(frame.data_ptr(), w, h, 3, 3 * w)
    det.Clear()
    del frame
    torch.cuda.empty_cache()
    assert any(x0 <= x < x0 + pw and y0 <= y < h for x, y, *_ in faces)
