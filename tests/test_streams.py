"""Executors on streams of their own share no scratch: what one launch leaves for the next belongs to their stream."""
import ctypes
import gc
import types
import weakref

import numpy as np
import pytest
import torch

from tsplit_b200 import _base, gpu_ops as ad, ndarray
from tsplit_b200.ops import _gpu as G
from tsplit_b200.runtime import cudagraph
from tsplit_b200.stream import Stream


def _rand(*shape, seed=0):
    t = torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
    torch.cuda.synchronize()                       # (read on other streams)
    return ndarray.from_tensor(t, ndarray.gpu(0))


def _image(*shape, seed=0):
    a = ndarray.empty(shape, ndarray.gpu(0), use_pool=False)
    a.t.copy_(_rand(*shape, seed=seed).t)
    torch.cuda.synchronize()
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
    torch.cuda.synchronize()
    _base.kernels().tsb_scratch_trim()             # (given-back buffers would be taken)
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


def _pointers(monkeypatch, shape, pads, stride, streams):
    """The calls of a stem's forward pass and filter gradient on each stream: [(entry, address of the packed image)]."""
    calls = []

    class Lib(object):
        def __getattr__(self, name):
            def entry(*args):
                at = {"tsb_pack_pixels": 1, "tsb_pack_pixel_rows": 1, "tsb_stem_wgrad": 0, "tsb_conv2d": 1}.get(name)
                calls.append((name, None if at is None else args[at].value))
                return 0
            return entry
    monkeypatch.setattr(G, "lib", lambda: Lib())
    def empty(shape, ctx, **kw):                  # channels last, as on a GPU
        t = torch.empty(shape)
        return ndarray.from_tensor(t if t.dim() != 4 else t.to(memory_format=torch.channels_last), ctx)
    monkeypatch.setattr(ndarray, "empty", empty)
    n, c, h, w, o, k = shape
    oh, ow = (h + 2 * pads - k) // stride + 1, (w + 2 * pads - k) // stride + 1
    x, f, y = (ndarray.empty(s, ndarray.cpu(0)) for s in ((n, c, h, w), (o, c, k, k), (n, o, oh, ow)))
    res, by_handle = [], {}
    for handle in streams:
        stream = by_handle.setdefault(handle, types.SimpleNamespace(handle=handle, buffers={}))
        for kind in (0, 2):
            G.conv2d(kind, x, f, y, pads, pads, stride, stream)
        res.append([c for c in calls if c[1] is not None])
        del calls[:]
    return res, sum(b[1].t.numel() for s in by_handle.values() for b in s.buffers.values() if isinstance(b, tuple))


@pytest.mark.parametrize("shape,pads,stride", [((4, 3, 64, 64, 16, 7), 3, 2), ((4, 3, 64, 64, 16, 7), 3, 1),
                                               ((4, 5, 64, 64, 16, 7), 3, 2)])
def test_packed_images_belong_to_a_stream(monkeypatch, shape, pads, stride):
    (first, second, again), _ = _pointers(monkeypatch, shape, pads, stride, (11, 12, 11))
    assert first == again and not {p for _, p in first} & {p for _, p in second}


def test_windows_take_the_room_of_the_packed_image(monkeypatch):
    (calls,), floats = _pointers(monkeypatch, (4, 3, 64, 64, 16, 7), 3, 2, (11,))
    assert [name for name, _ in calls] == ["tsb_pack_pixels", "tsb_conv2d", "tsb_pack_pixel_rows", "tsb_stem_wgrad"]
    assert len({p for _, p in calls}) == 1 and floats == 4 * 64 * (31 * 2 + 8) * 4          # the wider rows


@pytest.mark.parametrize("shape,stride", [((1, 3, 16, 16, 8, 3), 2), ((4, 3, 64, 64, 10, 3), 2), ((4, 3, 64, 64, 16, 9), 2)])
def test_nothing_is_packed_for_a_refusal(monkeypatch, shape, stride):
    """Images too small for the windows' tensor maps, filters of no whole 16 bytes, of nine taps."""
    (calls,), floats = _pointers(monkeypatch, shape, 1, stride, (11,))
    assert [name for name, _ in calls] == ["tsb_pack_pixels", "tsb_conv2d"] * 2
    assert floats == shape[0] * shape[2] * shape[3] * 4


@pytest.mark.parametrize("shape,stride,zeroed", [((4, 3, 64, 64, 16, 7), 2, 1), ((4, 5, 64, 64, 16, 7), 2, 2)])
def test_padding_is_zeroed_in_the_order_of_the_stream(monkeypatch, shape, stride, zeroed):
    """(Another stream's pass over a new buffer may come behind what this one has put there.)"""
    streams = []
    monkeypatch.setattr(torch.Tensor, "zero_", None)
    monkeypatch.setattr(G, "fill", lambda y, value, stream: streams.append((value, stream.handle)))
    _pointers(monkeypatch, shape, 3, stride, (11,))
    assert streams == [(0.0, 11)] * zeroed            # padded filters, and images of more than four channels


@pytest.mark.gpu
def test_buffers_are_given_back_with_their_stream():
    ctx = ndarray.gpu(0)
    x, f, y = _image(4, 3, 64, 64), _image(16, 3, 7, 7, seed=1), _image(4, 16, 32, 32)
    stream = Stream(ctx)
    other = Stream(ctx, torch_stream=stream.torch_stream)
    handle = weakref.ref(stream.buffers)
    G.conv2d(0, x, f, y, 3, 3, 2, stream)
    assert len(other.buffers) == 2 and Stream(ctx).buffers is not other.buffers
    want = y.t.clone()
    del stream
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    G.conv2d(0, x, f, y, 3, 3, 2, other)                       # the same ones
    assert torch.cuda.memory_allocated() == held
    del other
    assert handle() is None and held - torch.cuda.memory_allocated() >= 4 * 64 * 64 * 16
    torch.cuda.synchronize()
    assert torch.equal(y.t, want)


@pytest.mark.gpu
def test_scratch_of_a_finished_stream_is_for_the_next_one():
    """Handed on once the stream, and what was captured on it, has gone; another stream's stays its own."""
    ctx = ndarray.gpu(0)
    held = _base.kernels().tsb_scratch_bytes
    held.restype = ctypes.c_longlong
    torch.cuda.synchronize()
    gc.collect()
    _base.kernels().tsb_scratch_trim()
    first, other = Stream(ctx), Stream(ctx)
    want = [o.t.clone() for o in (_losses(first), torch.cuda.synchronize())[0]]
    graph = cudagraph.capture(first, lambda: None)
    del first
    before = held()
    _losses(other)
    torch.cuda.synchronize()
    assert held() > before                         # the graph may still be replayed
    del graph
    before = held()
    third = Stream(ctx)
    got = (_losses(third), torch.cuda.synchronize())[0]
    assert held() == before and all(torch.equal(g.t, w) for g, w in zip(got, want))
    assert (_losses(Stream(ctx)), torch.cuda.synchronize())[0] and held() > before


@pytest.mark.gpu
@pytest.mark.parametrize("executor", ["Executor", "microopExecutor"])
def test_first_step_behind_work_on_the_current_stream(executor):
    """Running statistics, step counter, padded operands and slots of a first step do not wait for one another by luck."""
    ctx, results = ndarray.gpu(0), []
    for busy in (False, True):
        r = np.random.default_rng(0)
        val = lambda *shape: (0.2 * r.standard_normal(shape)).astype(np.float32)
        x, y, w, s, b, wd = (ad.Variable(n, value=v) for n, v in (
            ("x", None), ("y", None), ("w", val(16, 5, 3, 3)), ("s", val(1, 16, 1, 1)), ("b", val(1, 16, 1, 1)), ("wd", val(1024, 12))))
        norm = ad.batch_normalization_op(ad.conv2d_op(x, w, padding=1, stride=2), s, b)
        drop = ad.dropout_op(norm, 0.7)
        drop.attrs["seed"] = 5
        loss = ad.softmaxcrossentropy_op(ad.matmul_op(ad.array_reshape_op(drop, (-1, 1024)), wd), y)
        grads = ad.gradients(loss, [w])
        feed = {x: ndarray.array(val(8, 5, 16, 16), ctx), y: ndarray.array(np.eye(12, dtype=np.float32)[np.arange(8)], ctx)}
        for v in (w, s, b, wd):
            v.tensor_value = ndarray.array(v.tensor_value, ctx)
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(200_000_000)                  # a tenth of a second
        ex = getattr(ad, executor)([loss, norm] + grads, ctx=ctx)
        results.append([o.t.clone() for _ in range(2) for o in ex.run(feed)])
        torch.cuda.synchronize()
        results[-1] += [norm.state[k].t.clone() for k in ("run_mean", "run_var")]
    assert all(torch.equal(p, q) for p, q in zip(*results))
