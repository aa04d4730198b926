"""The gate's training kernels at the sizes where their 32 x 16 pixel tiles end (one pixel more or less, odd
planes whose last row or column belongs to no cell, the smallest planes) against the float64 restatement,
and one Adam step against the device's own gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from compactcnncascade_b200 import gate  # noqa: E402
from oracle import gate_ref  # noqa: E402


def _data(n, w8, h8):
    rng = np.random.default_rng(1000 * w8 + h8)
    feat = rng.uniform(-2, 2, (n, h8, w8)).astype(np.float16)
    lab = (rng.random((n, 4, h8 // 2, w8 // 2)) < 0.1).astype(np.uint8)
    params = gate.init_params(w8 % 7)
    params[gate.B3:] = -1.5
    return feat, lab, params, gate.Dataset(torch.from_numpy(feat).cuda(), torch.from_numpy(lab).cuda(), int(lab.sum()))


@pytest.mark.parametrize("n,w8,h8", [(1, 2, 2), (2, 3, 5), (1, 31, 15), (1, 32, 16), (2, 33, 17), (1, 65, 34), (1, 64, 1 + 2 * 16), (7, 240, 135)])
def test_gradient_at_tile_edges(n, w8, h8):
    feat, lab, params, ds = _data(n, w8, h8)
    loss, g = gate.gradient(params, ds, 12.0)
    want_loss, want = gate_ref.loss_and_grad(params, feat.astype(np.float64), lab, 12.0, fp16=True)
    assert abs(loss - want_loss) <= 1e-4 * abs(want_loss)
    # the bounds of the gradient's other test: fp32 sums and rare flips of an activation's binary16 rounding
    assert np.linalg.norm(g - want) <= 2e-3 * np.linalg.norm(want)
    assert np.allclose(g, want, rtol=2e-2, atol=2e-3 * np.abs(want).max())
    again = gate.gradient(params, ds, 12.0)
    assert again[0] == loss and np.array_equal(again[1], g)


def test_adam_steps_follow_the_gradient():
    """Two steps of training equal Adam, in float64, on the gradients the device gives at the same parameters."""
    feat, lab, params, ds = _data(4, 40, 30)
    half = [gate.Dataset(ds.feat[k:k + 2].contiguous(), ds.labels[k:k + 2].contiguous(), 0) for k in (0, 2)]
    got, losses = gate.train(ds, params, epochs=1, batch=2, lr=3e-3, pos_weight=12.0)
    first, l0 = gate.train(half[0], params, epochs=1, batch=2, lr=3e-3, pos_weight=12.0)
    g = [gate.gradient(params, half[0], 12.0)[1].astype(np.float64), gate.gradient(first, half[1], 12.0)[1].astype(np.float64)]
    l1 = gate.gradient(first, half[1], 12.0)[0]
    m = v = np.zeros(700)
    p = params.astype(np.float64)
    for k in range(2):
        m, v = 0.9 * m + 0.1 * g[k], 0.999 * v + 0.001 * g[k] ** 2
        p = p - 3e-3 * (m / (1 - 0.9 ** (k + 1))) / (np.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
        # fp32: the moments and bias corrections carry a few ulps (1 - 0.999 in fp32 is off by 5e-5 relative,
        # which the square root halves)
        assert np.allclose(first if k == 0 else got, p, rtol=1e-5, atol=3e-3 * 1e-4)
    assert abs(losses[0] - (l0[0] + l1) / 2) <= 1e-6 * abs(losses[0])
