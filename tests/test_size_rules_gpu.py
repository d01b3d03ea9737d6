"""Kernels chosen by size: each rule at the edges of its range, against 64-bit torch."""
import numpy as np
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
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda")


def _stream():
    from tsplit_b200.stream import current_stream
    return current_stream(ndarray.gpu(0))


# one split; a ragged channel block with eight splits; padded windows that overlap; rows of one pixel; the widest
@pytest.mark.parametrize("n,c,h,w,kh,kw,pad,stride", [(2, 4, 6, 6, 6, 6, 0, 6), (1, 36, 57, 57, 57, 57, 0, 57),
                                                      (2, 8, 20, 23, 9, 9, 4, 3), (3, 12, 40, 1, 40, 1, 0, 40),
                                                      (1, 64, 130, 130, 130, 130, 0, 130)])
def test_average_pool_large_windows(n, c, h, w, kh, kw, pad, stride):
    x = _rand(n, c, h, w) + 1
    ref = torch.nn.functional.avg_pool2d(x.double(), (kh, kw), stride, pad)
    y = _arr(torch.zeros(ref.shape, device="cuda"))
    G.pool(1, _arr(x), y, kh, kw, pad, stride, _stream())
    # sums of at most a few hundred terms per lane and pairwise joins: far below 1e-5 of the mean magnitude
    torch.testing.assert_close(y.t.double(), ref, rtol=1e-5, atol=1e-5)
