"""Executors on streams of their own share no scratch: what one launch leaves for the next belongs to their stream."""
import ctypes

import pytest
import torch

from tsplit_b200 import _base, ndarray
from tsplit_b200.ops import _gpu as G
from tsplit_b200.stream import Stream


def _rand(*shape, seed=0):
    return ndarray.from_tensor(torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda"), ndarray.gpu(0))


def _image(*shape, seed=0):
    a = ndarray.empty(shape, ndarray.gpu(0), use_pool=False)
    a.t.copy_(_rand(*shape, seed=seed).t)
    return a


def _losses(stream):
    x, lab, g, loss, dx = _rand(64, 10), _rand(64, 10, seed=1), _rand(1, seed=2), _rand(1), _rand(64, 10)
    assert G.softmax_ce_both(x, lab, g, loss, dx, stream)
    return loss, dx


def _batch_norm(stream):
    x, y, scale, bias, *stats = [_image(2, 64, 9, 9, seed=i) for i in range(2)] + [_rand(64, seed=i) for i in range(6)]
    G.bn_forward(x, scale, bias, y, *stats, 0.9, 0.01, False, stream)
    return [y] + stats


def _layer_norm_grad(stream):
    dy, x, dx = (_rand(300, 96, seed=i) for i in range(3))
    small = [_rand(n, seed=n + i) for i, n in enumerate((96, 300, 300, 96, 96))]
    G.layer_norm_grad(dy, x, *small[:3], dx, *small[3:], stream)
    return [dx] + small[3:]


def _column_sums(stream):
    x, y = _rand(5000, 64), _rand(64)
    G.reduce_sum(x.ptr, x.shape, x.strides, [0], y, stream)
    return y,


def _wide_max_pool_grad(stream):
    x, y, dy, dx = _image(2, 8, 20, 20), _image(2, 8, 16, 16, seed=1), _image(2, 8, 16, 16, seed=2), _image(2, 8, 20, 20)
    G.pool_grad(0, x, y, dy, dx, 5, 5, 0, 1, stream)
    return dx,


@pytest.mark.gpu
@pytest.mark.parametrize("run", [_losses, _batch_norm, _layer_norm_grad, _column_sums, _wide_max_pool_grad])
def test_each_stream_has_scratch_of_its_own(run):
    held = _base.kernels().tsb_scratch_bytes
    held.restype = ctypes.c_longlong
    outs = []
    for _ in range(2):
        handle = ctypes.c_void_p()                 # (a new one: torch's streams come from a pool)
        assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
        stream = Stream(ndarray.gpu(0), torch_stream=torch.cuda.ExternalStream(handle.value))
        torch.cuda.synchronize()
        before = held()
        outs.append([o.t.clone() for o in (run(stream), torch.cuda.synchronize())[0]])
        assert held() > before
    assert all(torch.equal(a, b) for a, b in zip(*outs))
