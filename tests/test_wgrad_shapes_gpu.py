"""Weight gradients at every row shape of the weight-gradient kernel's K-step.

A step is one row segment of 128 pixels above width 64, else 128 / Wp rows of Wp = 16, 32, 48 or 64 pixels; the
four levels of a network of width w run at w, w/2, w/4 and w/8.  The sizes below reach each shape with ragged
widths, heights that leave part of a step's rows outside the image, fewer steps than SMs, and more.
"""
import numpy as np
import pytest

import lumina

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
F = torch.nn.functional

import unet_ref  # noqa: E402


def _grads(model, flat, noisy, clean, dtype):
    m = unet_ref.load_flat(model, flat).to(dtype)
    out = unet_ref.forward_bf16(m, torch.from_numpy(noisy), dtype=dtype)
    F.l1_loss(out, torch.from_numpy(clean).to(dtype)).backward()
    return [(k, p.grad.double().numpy().ravel()) for k, p in m.named_parameters()]


@pytest.mark.parametrize("n,h,w", [(4, 24, 40), (4, 16, 72), (4, 16, 64), (3, 40, 128), (1, 64, 136), (5, 56, 96)])
def test_gradients_at_every_row_shape(n, h, w):
    """Against autograd through the BF16-emulated restatement in FP64; per tensor the relative L2 error stays
    within 3x the emulation's own FP32-to-FP64 noise + 1%, the cosine above 0.998."""
    flat = unet_ref.make_params(21, unet_ref.UNetRef())
    net = lumina.UNet()
    net.set_params(flat)
    rng = np.random.default_rng(4)
    noisy = rng.uniform(0.3, 0.7, (n, 3, h, w)).astype(np.float32)
    clean = np.full_like(noisy, -1.0)  # below every prediction: no sign of the L1 loss hangs on a rounding
    dx, dt = torch.from_numpy(noisy).cuda(), torch.from_numpy(clean).cuda()
    _, g = net.loss_grad(dx.data_ptr(), dt.data_ptr(), n, h, w)
    _, again = net.loss_grad(dx.data_ptr(), dt.data_ptr(), n, h, w)
    assert np.array_equal(g, again)  # the chunks are added in a fixed order
    g64 = _grads(unet_ref.UNetRef(), flat, noisy, clean, torch.float64)
    g32 = _grads(unet_ref.UNetRef(), flat, noisy, clean, torch.float32)
    off = 0
    for (k, want), (_, low) in zip(g64, g32):
        got = g[off:off + want.size].astype(np.float64)
        off += want.size
        norm = np.linalg.norm(want) + 1e-30
        rel, floor = np.linalg.norm(got - want) / norm, np.linalg.norm(low - want) / norm
        cos = np.dot(got, want) / (np.linalg.norm(got) * norm + 1e-30)
        assert cos > 0.998 and rel <= 3 * floor + 0.01, (k, cos, rel, floor)
