"""Calls ordered on a caller's stream: when that stream cannot be ordered against, the call says so and queues nothing.
The stream used here is one whose capture was ended by a wait on it, which CUDA answers with an error and until the
capture is closed refuses events on the stream."""
import ctypes as C

import numpy as np
import pytest

import lumina
from lumina import _ffi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class InvalidatedCapture:
    def __enter__(self):
        self.cu = C.CDLL("libcuda.so.1")
        self.stream = torch.cuda.Stream()
        h = C.c_void_p(self.stream.cuda_stream)
        assert self.cu.cuStreamBeginCapture_v2(h, 2) == 0  # relaxed: other streams are not concerned
        assert self.cu.cuStreamSynchronize(h) == 900  # CUDA_ERROR_STREAM_CAPTURE_UNSUPPORTED
        return self.stream.cuda_stream

    def __exit__(self, *exc):
        graph = C.c_void_p()
        self.cu.cuStreamEndCapture(C.c_void_p(self.stream.cuda_stream), C.byref(graph))


def _frame(r, cam, stream):
    c, o, d = cam.to_c(), _ffi.LgRenderOpts(2, 1, 0, 0), C.c_void_p()
    rc = _ffi.lib().lg_render_device(r._h, C.byref(c), C.byref(o), C.c_void_p(stream), None, C.byref(d), None)
    return rc, d.value


def _read(ptr, n):
    out = np.empty(n, np.float32)
    assert C.CDLL("libcuda.so.1").cuMemcpyDtoH_v2(C.c_void_p(out.ctypes.data), C.c_uint64(ptr), C.c_size_t(4 * n)) == 0
    return out


def test_render_device(box_scene):
    cam = box_scene.camera
    other = cam.look_at([3, 3, 2.5], [0, 0, 1])
    n = int(cam.width) * int(cam.height) * 3
    with lumina.Renderer(0) as r:
        r.set_scene(box_scene)
        rc, ptr = _frame(r, cam, torch.cuda.Stream().cuda_stream)
        torch.cuda.synchronize()
        first = _read(ptr, n)
        assert rc == 0 and first.any()
        with InvalidatedCapture() as stream:
            rc, _ = _frame(r, other, stream)
            assert rc == _ffi.LG_ERR_CUDA
        torch.cuda.synchronize()
        assert np.array_equal(_read(ptr, n), first)  # the refused frame was not rendered
        rc, ptr = _frame(r, other, torch.cuda.Stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0 and np.array_equal(_read(ptr, n), r.render(camera=other, spp=2, bounces=1)["accum"].ravel())


def test_unet_forward_device():
    net = lumina.UNet()
    net.set_params(np.random.default_rng(5).normal(0, 0.05, net.n_params).astype(np.float32))
    x = torch.rand((1, 3, 16, 24), device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    with InvalidatedCapture() as stream:
        with pytest.raises(lumina.LuminaError) as e:
            net.forward_device(x.data_ptr(), 1, 16, 24, y.data_ptr(), stream)
        assert e.value.code == _ffi.LG_ERR_CUDA
    torch.cuda.synchronize()
    assert not y.any()
    net.forward_device(x.data_ptr(), 1, 16, 24, y.data_ptr(), torch.cuda.Stream().cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), net.forward(x.cpu().numpy()))
