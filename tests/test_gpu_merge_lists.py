"""The one-warp merge of long lists against the restatement of Merger (oracle/facial_ref.py): NMS of random boxes
(boxes, their order, scores) and detection behind many earlier detections, around the 32 boxes of a step."""
import ctypes

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


@pytest.fixture(scope="module")
def handle():
    cp, ca, h = _capi.CnnParam(), _capi.CnnAdvancedParam(), ctypes.c_void_p()
    L = _capi.lib()
    L.ccnn_cnn_default_params(ctypes.byref(cp), ctypes.byref(ca))
    cp.max_image_width, cp.max_image_height, cp.min_obj_height, cp.max_obj_height, cp.scale_factor = 640, 480, 30, 240, 1.1
    ca.detect_precision = 3
    _capi.check(L.ccnn_cnn_create(ctypes.byref(cp), ctypes.byref(ca), None, ctypes.byref(h)), "ccnn_cnn_create")
    yield h
    L.ccnn_destroy(h)


def _boxes(n, seed, size):
    rng = np.random.default_rng(seed)
    return [(int(x), int(y), int(w), int(h), float(np.float32(s))) for x, y, w, h, s in
            zip(rng.integers(0, 560, n), rng.integers(0, 400, n), rng.integers(size // 2, size, n), rng.integers(size // 2, size, n), rng.random(n))]


def _list(boxes):
    return (_capi.Detection * max(1, len(boxes)))(*[_capi.Detection(*b, 0.5, 1, 3) for b in boxes])


def _corners(boxes):
    return [(x, y, x + w, y + h, s) for x, y, w, h, s, *_ in boxes]


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 97, 700])
@pytest.mark.parametrize("size", [40, 200])
def test_nms(handle, n, size):
    boxes = _boxes(n, 7 * n + size, size)
    out, k = (_capi.Detection * n)(), ctypes.c_int()
    _capi.check(_capi.lib().ccnn_cnn_nms(handle, _list(boxes), n, out, n, ctypes.byref(k)), "ccnn_cnn_nms")
    want, _ = facial_ref.merger(_corners(boxes), 0.5, False)
    assert [(d.x, d.y, d.x + d.width, d.y + d.height, d.score) for d in out[:k.value]] == want


@pytest.mark.parametrize("n", [1, 30, 33, 300])
def test_behind_earlier_detections(handle, n):
    img, _ = ccnn.synth_frame(640, 480, 5, 6, 40, 120)
    prior = _boxes(n, n, 120)
    im, out, k = _capi.Image(640, 480, 3, img.ctypes.data, 1920), (_capi.Detection * 1000)(), ctypes.c_int()
    L = _capi.lib()
    _capi.check(L.ccnn_cnn_detect(handle, ctypes.byref(im), _list(prior), n, out, 1000, ctypes.byref(k)), "ccnn_cnn_detect")
    raw, m = (_capi.Detection * 4096)(), ctypes.c_int()
    _capi.check(L.ccnn_inspect_raw_detections(handle, raw, 4096, ctypes.byref(m)), "ccnn_inspect_raw_detections")
    raw = [(d.x, d.y, d.width, d.height, d.score, d.scale) for d in raw[m.value - 1::-1]]
    assert len(raw) > 4
    order = orc.sort_perm([r[5] for r in raw])
    clusters, _ = facial_ref.merger(_corners([raw[i] for i in order]), 0.5, False)
    want, _ = facial_ref.merger(_corners(prior) + clusters, 0.2, True)
    assert [(d.x, d.y, d.x + d.width, d.y + d.height, d.score) for d in out[:k.value]] == want
