"""Filter gradient of strided few-channel stems by TMA windows: the bits of the gathering path."""
import ctypes

import pytest
import torch

from tsplit_b200 import _base, ndarray
from tsplit_b200.ops import _gpu as G

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def _arr(t):
    a = ndarray.empty(tuple(t.shape), ndarray.gpu(0), use_pool=False)
    a.t.copy_(t)
    return a


def _stream():
    from tsplit_b200.stream import current_stream
    return current_stream(ndarray.gpu(0))


# the 7x7 stem; odd sizes whose windows end behind the image; eight taps and no padding; filters of no 32 channels, of more
# than one row tile; one and two channels; a stride that skips pixels; output rows shorter than a k-block, a partial last one
@pytest.mark.parametrize("n,c,h,w,o,kh,kw,pad,stride", [
    (4, 3, 64, 64, 64, 7, 7, 3, 2), (2, 3, 75, 61, 32, 3, 3, 0, 2), (2, 1, 96, 96, 64, 8, 8, 0, 2), (3, 3, 57, 70, 20, 5, 7, 2, 2),
    (1, 2, 130, 90, 160, 7, 3, 3, 3), (4, 3, 100, 33, 64, 3, 8, 1, 5), (5, 3, 41, 60, 48, 7, 7, 6, 2)])
def test_filter_gradient(n, c, h, w, o, kh, kw, pad, stride):
    oh, ow = (h + 2 * pad - kh) // stride + 1, (w + 2 * pad - kw) // stride + 1
    x, dy = _arr(_rand(n, c, h, w)), _arr(_rand(n, o, oh, ow, seed=1))
    dw = _arr(torch.full((o, c, kh, kw), 7.0, device="cuda"))
    assert G._strided_stem_wgrad(x, dw, dy, pad, pad, stride, _stream())
    x4, want = _arr(torch.zeros((n, 4, h, w), device="cuda")), _arr(torch.zeros((o, 4, kh, kw), device="cuda"))
    x4.t[:, :c] = x.t
    lib, ptr = _base.kernels(), lambda a: ctypes.c_void_p(a.ptr)
    rc = lib.tsb_conv2d(2, ptr(x4), ptr(want), ptr(dy), n, 4, h, w, o, kh, kw, oh, ow, pad, pad, stride,
                        G._s(_stream()))
    torch.cuda.synchronize()
    assert rc == 0
    assert torch.equal(dw.t, want.t[:, :c])
    assert lib.tsb_device_status(ctypes.c_void_p(0)) == 0


def test_small_images_take_the_gathering_path():
    x, dy = _arr(_rand(1, 3, 16, 16)), _arr(_rand(1, 8, 8, 8, seed=1))
    dw = _arr(torch.zeros((8, 3, 3, 3), device="cuda"))
    assert not G._strided_stem_wgrad(x, dw, dy, 1, 1, 2, _stream())
    G.conv2d(2, x, dw, dy, 1, 1, 2, _stream())
    ref = torch.nn.grad.conv2d_weight(x.t.double(), dw.t.shape, dy.t.double(), stride=2, padding=1)
    assert (dw.t.double() - ref).norm() < 2e-3 * ref.norm()                   # operands of 10 bits
