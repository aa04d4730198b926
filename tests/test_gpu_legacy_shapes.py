"""The legacy (format 1.0) forward pass over the network shapes that the format admits (map counts, max and
average pooling, third-layer kernels, both hidden layers) and the image sizes where its 32 x 8 tiles end,
against the float32 restatement bit for bit. The networks are seeded random ones."""
import ctypes
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from compactcnncascade_b200 import _capi  # noqa: E402
from oracle import legacy_ref  # noqa: E402


def _model(path, m0, max_pool, kw, kh, fc, hl):
    rng = np.random.default_rng(100 * m0 + 10 * kw + kh + max_pool)
    maps = [m0, 2 * m0, 4 * m0]
    ks = [(4, 4), (3, 3), (kw, kh)]

    def f(n, scale=1.0):
        return (rng.standard_normal(n) * scale).astype("<f4").tobytes()

    blob = struct.pack("<fBiii", 1.0, max_pool, 8, 8, 3) + struct.pack("<iii", *maps)
    for m, (w, h), s in zip(maps, ks, (0.004, 0.3, 0.2)):
        blob += struct.pack("<ii", w, h) + f(m * w * h, s)
    blob += struct.pack("<f", 1.7159)
    for m in maps:
        blob += f(3 * m)
    blob += struct.pack("<Bi", fc, hl) + f(hl * maps[2] if fc else hl, 0.5) + f(hl) + f(hl, 0.5) + f(1)
    path.write_bytes(blob)
    return str(path)


@pytest.mark.parametrize("m0,max_pool,kw,kh,fc,hl", [(2, 1, 5, 6, 0, 16), (3, 0, 5, 6, 0, 24), (4, 1, 5, 6, 0, 32), (4, 0, 7, 8, 1, 10), (5, 1, 6, 5, 0, 40),
                                                     (6, 0, 7, 8, 0, 48), (6, 0, 7, 8, 1, 48), (6, 1, 10, 3, 1, 5), (8, 1, 5, 6, 1, 64), (8, 0, 7, 8, 0, 64)])
@pytest.mark.parametrize("ow,oh,extra,pad", [(1, 1, 0, 0), (32, 8, 3, 1), (33, 9, 1, 0), (31, 17, 2, 3), (100, 41, 0, 0)])
def test_forward(tmp_path, m0, max_pool, kw, kh, fc, hl, ow, oh, extra, pad):
    path = _model(tmp_path / "m.bin", m0, max_pool, kw, kh, fc, hl)
    w, h = ((ow + kw - 1) * 2 + 2) * 2 + 3 + extra, ((oh + kh - 1) * 2 + 2) * 2 + 3 + (extra * 3) % 4
    img = np.random.default_rng(ow + oh).uniform(0, 255, (h, w)).astype(np.float32)
    want = legacy_ref.forward(legacy_ref.load(path), img)
    assert want.shape == (oh, ow)
    buf = torch.zeros((h, w + pad), dtype=torch.float32, device="cuda")
    buf[:, :w] = torch.from_numpy(img).cuda()
    out = torch.zeros(ow * oh, dtype=torch.float32, device="cuda")
    gw, gh = ctypes.c_int(), ctypes.c_int()
    st = _capi.lib().ccnn_legacy_net_forward(path.encode(), buf.data_ptr(), w, h, (w + pad) * 4, out.data_ptr(), out.numel(), ctypes.byref(gw),
                                             ctypes.byref(gh), None)
    assert st == _capi.OK, _capi.last_error()
    assert (gw.value, gh.value) == (ow, oh)
    assert np.array_equal(out.cpu().numpy().reshape(oh, ow).view(np.uint32), want.view(np.uint32))
