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
@pytest.mark.parametrize("n,c,h,w,kh,kw,pad,stride", [(2, 4, 8, 8, 8, 8, 0, 8), (1, 36, 57, 57, 57, 57, 0, 57),
                                                      (2, 8, 20, 23, 9, 9, 4, 3), (3, 12, 70, 1, 70, 1, 0, 70),
                                                      (1, 64, 130, 130, 130, 130, 0, 130)])
def test_average_pool_large_windows(n, c, h, w, kh, kw, pad, stride):
    x = _rand(n, c, h, w) + 1
    ref = torch.nn.functional.avg_pool2d(x.double(), (kh, kw), stride, pad)
    y = _arr(torch.zeros(ref.shape, device="cuda"))
    G.pool(1, _arr(x), y, kh, kw, pad, stride, _stream())
    # sums of at most a few hundred terms per lane and pairwise joins: far below 1e-5 of the mean magnitude
    torch.testing.assert_close(y.t.double(), ref, rtol=1e-5, atol=1e-5)


# a tensor below one vector, a vector's remainder, one tile less, exactly and more than one element, and several tiles;
# views that start 4 bytes in take the scalar form
@pytest.mark.parametrize("n", [1, 3, 2047, 2048, 2049, 7 * 2048 + 5])
@pytest.mark.parametrize("shift", [0, 1])
def test_streaming_kernels_cover_the_tensor_once(n, shift):
    a, b = _rand(n + shift)[shift:], _rand(n + shift, seed=1)[shift:]
    ctx = ndarray.gpu(0)
    x, z = ndarray.from_tensor(a, ctx), ndarray.from_tensor(b, ctx)
    out = torch.full((n + shift + 8,), 7.0, device="cuda")
    y = ndarray.from_tensor(out[shift:n + shift], ctx)
    for run, ref in ((lambda: G.unary(G.UN_MULC, x, y, _stream(), alpha=3.0), a * 3),
                     (lambda: G.fill(y, 2.5, _stream()), torch.full((n,), 2.5, device="cuda")),
                     (lambda: G.binary(G.BIN_ADD, x, z, y, _stream()), a + b)):
        run()
        assert torch.equal(y.t, ref)                    # one rounding each: the same bits
        assert torch.all(out[n + shift:] == 7) and torch.all(out[:shift] == 7)


def test_optimizer_tiles_of_many_tensors():
    sizes = [1, 2047, 2048, 2049, 5, 3 * 2048, 1000] * 9 + [4097]         # 64 tensors of one launch
    ctx = ndarray.gpu(0)
    ps, gs, vs = ([ndarray.from_tensor(_rand(n, seed=k + 100 * j), ctx) for k, n in enumerate(sizes)] for j in range(3))
    want = [(0.9 * v.t - 0.01 * g.t, p.t.clone()) for p, g, v in zip(ps, gs, vs)]
    G.optimizer_step(1, ps, gs, vs, None, [0.01, 0.9], _stream())
    for (v1, p0), p, v in zip(want, ps, vs):
        # two products, an addition and an update in fp32, contracted or not: a few units in the last place of values < 8
        torch.testing.assert_close(v.t, v1, rtol=0, atol=2e-6)
        torch.testing.assert_close(p.t, p0 + v1, rtol=0, atol=4e-6)
