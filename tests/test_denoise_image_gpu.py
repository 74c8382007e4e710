"""8-bit frames denoised on the device (lg_unet_denoise_rgb8): the same bytes as the host conversion around
the FP32 forward pass, at sizes with and without padding."""
import numpy as np
import pytest

import lumina

pytestmark = pytest.mark.gpu


def _host(net, planes):
    """tools/denoise.py:34-52 in numpy around UNet.forward."""
    x = np.concatenate([p.astype(np.float32) / 255.0 for p in planes], axis=2)
    h, w = x.shape[:2]
    x = np.pad(x, ((0, -h % 8), (0, -w % 8), (0, 0)), mode="edge")
    y = net.forward(x.transpose(2, 0, 1)[None])[0].transpose(1, 2, 0)[:h, :w]
    return (np.clip(y, 0.0, 1.0) * 255.0 + 0.5).astype(np.uint8)


@pytest.mark.parametrize("in_ch", [3, 12])
@pytest.mark.parametrize("h,w", [(1, 1), (8, 16), (9, 17), (37, 130), (96, 265)])
def test_same_bytes_as_host_conversion(in_ch, h, w):
    rng = np.random.default_rng(h * 1000 + w)
    net = lumina.UNet(in_ch=in_ch)
    net.set_params(rng.normal(0, 0.05, net.n_params).astype(np.float32))
    planes = [rng.integers(0, 256, (h, w, 3), dtype=np.uint8) for _ in range(in_ch // 3)]
    assert np.array_equal(net.denoise_rgb8(*planes), _host(net, planes))


def test_views_and_other_types():
    """A non-contiguous view, and an image that is not 8-bit, give what the host conversion gives."""
    rng = np.random.default_rng(1)
    net = lumina.UNet()
    net.set_params(rng.normal(0, 0.05, net.n_params).astype(np.float32))
    img = rng.integers(0, 256, (40, 60, 3), dtype=np.uint8)
    view = img[::2, ::-1]
    assert np.array_equal(net.denoise_rgb8(view), _host(net, [view]))
    assert np.array_equal(net.denoise_rgb8(img.astype(np.uint16)), _host(net, [img]))
