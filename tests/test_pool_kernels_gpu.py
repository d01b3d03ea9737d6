"""Pooling kernels of small windows and of windows that do not overlap, and the pixel packing, at the edges of their rules."""
import pytest
import torch

from tsplit_b200 import ndarray
from tsplit_b200.ops import _gpu as G

pytestmark = pytest.mark.gpu


def _arr(t, channels_last=None):
    a = ndarray.empty(tuple(t.shape), ndarray.gpu(0), use_pool=False, channels_last=channels_last)
    a.t.copy_(t)
    return a


def _rand(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def _stream():
    from tsplit_b200.stream import current_stream
    return current_stream(ndarray.gpu(0))


# one output; a last block of one thread; padding on all sides; odd sizes that leave a remainder; windows that overlap
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("n,c,h,w,k,pad,stride", [(1, 4, 2, 2, 2, 0, 2), (1, 4, 3, 3, 3, 0, 3), (1, 4, 32, 514, 2, 0, 2),
                                                  (2, 36, 9, 13, 3, 1, 2), (3, 20, 7, 8, 3, 1, 1), (2, 8, 15, 5, 2, 1, 1)])
def test_forward_of_small_windows(kind, n, c, h, w, k, pad, stride):
    x = _rand(n, c, h, w) - 1                         # mostly negative: padding must not take part in a maximum
    ref = (torch.nn.functional.max_pool2d if kind == 0 else torch.nn.functional.avg_pool2d)(x.double(), k, stride, pad)
    y = _arr(torch.zeros(ref.shape, device="cuda"))
    G.pool(kind, _arr(x), y, k, k, pad, stride, _stream())
    if kind == 0:
        assert torch.equal(y.t.double(), ref)
    else:                                             # at most nine terms: 9 * 2^-24 of their magnitudes
        torch.testing.assert_close(y.t.double(), ref, rtol=0, atol=9 * 2 ** -24 * x.abs().max().item())


# a channel vector that divides a block and one that does not, more channels than a block's threads; one window, several,
# a remainder of rows and columns that none covers, windows smaller than their stride, a row of many pixels
@pytest.mark.parametrize("n,c,h,w,kh,kw,stride", [(2, 4, 5, 5, 5, 5, 5), (1, 20, 17, 17, 17, 17, 17), (2, 1028, 3, 4, 3, 4, 4),
                                                  (3, 12, 13, 11, 4, 4, 4), (2, 8, 13, 11, 3, 2, 5), (1, 64, 4, 700, 4, 4, 4)])
def test_average_gradient_without_overlap(n, c, h, w, kh, kw, stride):
    x = _rand(n, c, h, w).double().requires_grad_()
    y = torch.nn.functional.avg_pool2d(x, (kh, kw), stride)
    dy = _rand(*y.shape, seed=1)
    ref, = torch.autograd.grad(y, x, dy.double())
    dx = _arr(torch.full((n, c, h, w), 7.0, device="cuda"))
    G.pool_grad(1, None, None, _arr(dy), dx, kh, kw, 0, stride, _stream())
    torch.testing.assert_close(dx.t.double(), ref, rtol=2 ** -22, atol=0)       # one product by a rounded 1 / (kh * kw)


@pytest.mark.parametrize("n,c,h,w", [(1, 1, 1, 1), (1, 3, 32, 32), (3, 2, 11, 31), (1, 3, 5, 205), (2, 3, 64, 64)])
def test_pixels_of_four_channels(n, c, h, w):
    """One pixel; exactly a block; one pixel more than a block; other remainders."""
    x = _arr(_rand(n, c, h, w))
    y = _arr(torch.full((n, 4, h, w), 7.0, device="cuda"))
    G._to_pixels(x, y, _stream())
    assert torch.equal(y.t[:, :c], x.t) and not y.t[:, c:].any()


# windows of 3 x 3 two apart: one pixel, tiles cut in both axes and at a window's middle, a ragged channel block, rows that no
# window reaches; many ties, and values below any finite one
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("n,c,h,w", [(1, 4, 3, 3), (2, 36, 16, 33), (1, 8, 15, 18), (2, 4, 34, 47), (3, 68, 4, 5)])
def test_max_gradient_of_3x3_windows(n, c, h, w, pad):
    from tsplit_b200.ops.pool import np_max_pool_grad
    x = torch.round(_rand(n, c, h, w) * 2) / 2
    x[x < -0.75] = -float("inf")
    y = torch.nn.functional.max_pool2d(x, 3, 2, pad)
    dy = torch.round(_rand(*y.shape, seed=1) * 8) / 8                # sums of four eighths are exact
    dx = _arr(torch.full((n, c, h, w), 7.0, device="cuda"))
    G.pool_grad(0, _arr(x), _arr(y), _arr(dy), dx, 3, 3, pad, 2, _stream())
    # (the oracle pads with -inf, which must not tie with a place inside)
    low = torch.where(torch.isinf(x), torch.full_like(x, -1e9), x).cpu().numpy()
    want = np_max_pool_grad(low, None, dy.cpu().numpy(), 3, 3, pad, 2)
    assert torch.equal(dx.t.cpu(), torch.from_numpy(want))
