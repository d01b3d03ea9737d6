"""A loss that waits for its gradient: the plan on the host, the kernels on the GPU against the separate ones."""

import numpy as np
import pytest
import torch

import test_step_plan as base
from tsplit_b200 import gpu_ops as ad, ndarray, optimizer
from tsplit_b200.ops import _gpu as G


def _both(calls):
    def run(logits, labels, g, loss, dx, stream):
        calls.append("dense")
        x, t = logits.numpy_view(), labels.numpy_view()
        p = np.exp(x - x.max(1, keepdims=True))
        p /= p.sum(1, keepdims=True)
        loss.numpy_view()[...] = np.mean(-(t * np.log(p)).sum(1))
        dx.numpy_view()[...] = (p - t) * g.numpy_view() / x.shape[0]
        return True

    def smooth(logits, ids, on, off, g, loss, dx, stream):
        calls.append("ids")
        assert base._smooth(False, True)(logits, ids, on, off, loss, stream)
        return base._smooth(True, True)(logits, ids, on, off, g, dx, stream)
    return run, smooth


def _net(smoothed, extra):
    def build():
        r = np.random.default_rng(0)
        x, w, y = (ad.Variable(n) for n in "xwy")
        logits = ad.matmul_op(x, w)
        feed = {x: r.standard_normal((6, 8), np.float32), w: r.standard_normal((8, 12), np.float32)}
        if smoothed:
            labels = ad.addbyconst_op(ad.mul_byconst_op(ad.one_hot_op(y, 12), 0.9), 0.01)
            feed[y] = np.array([0, 3, 11, 5, 5, 2], np.float32)
        else:
            labels = y
            feed[y] = np.eye(12, dtype=np.float32)[[0, 3, 11, 5, 5, 2]]
        loss = ad.softmaxcrossentropy_op(logits, labels)
        total = ad.mul_byconst_op(loss, 2.0) if extra else loss          # its value is read before the gradient
        return [total] + ad.gradients(total, [w, x]), feed
    return build


@pytest.mark.parametrize("smoothed", [False, True])
@pytest.mark.parametrize("taken", [False, True])
def test_one_pass_for_both(monkeypatch, smoothed, taken):
    calls = []
    if taken:
        dense, ids = _both(calls)
        monkeypatch.setattr(G, "softmax_ce_both", dense)
        monkeypatch.setattr(G, "softmax_ce_both_smooth", ids)
    plan = base._compare(monkeypatch, _net(smoothed, False), steps=2)
    assert len(plan.both) == 1 and calls == (["ids" if smoothed else "dense"] * 2 if taken else [])


def test_a_loss_that_is_read_is_not_late(monkeypatch):
    assert not base._compare(monkeypatch, _net(False, True)).both


def test_a_loss_does_not_wait_for_a_gradient_behind_an_update(monkeypatch):
    """Its labels are a variable that an optimizer trains between the two."""
    r = np.random.default_rng(0)
    xv, tv, lv = (r.standard_normal((6, 12)).astype(np.float32) for _ in range(3))
    dense, _ = _both([])
    monkeypatch.setattr(G, "softmax_ce_both", dense)

    def build():
        x, t, lab = ad.Variable("x"), ad.Variable("t"), ad.Variable("lab", value=np.abs(lv))
        loss = ad.softmaxcrossentropy_op(x, lab)
        diff = lab + ad.opposite_op(t)
        train = optimizer.SGDOptimizer(0.1).minimize(ad.reduce_sum_op(ad.mul_op(diff, diff), [0, 1]), [lab])
        return [loss, train] + ad.gradients(loss, [x]), {x: xv, t: tv}
    assert not base._compare(monkeypatch, build, steps=2).both


# a row of a few classes, more than a thread keeps, long rows: from L2, staged in shared memory, too long for that; ids
# outside the classes and masked classes
@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1, 10), (64, 10), (130, 1000), (33, 1021), (7, 5000), (5, 8192), (300, 8192), (160, 32000),
                                       (3, 51204), (2500, 512)])
def test_bits_of_separate_kernels(rows, cols):
    ctx = ndarray.gpu(0)
    from tsplit_b200.stream import current_stream
    st = current_stream(ctx)
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = 3 * torch.randn((rows, cols), device="cuda", generator=gen)
    x[:, 1::7] = -1e9
    x[0, 3] = torch.finfo(torch.float32).min
    ids = torch.randint(0, cols, (rows,), device="cuda", generator=gen).float()
    ids[0] = cols if rows > 1 else 0
    lab = torch.rand((rows, cols), device="cuda", generator=gen)
    lab[x < -1e8] = 0
    a = lambda t: ndarray.from_tensor(t, ctx)
    g = a(torch.full((1,), 0.5, device="cuda"))
    want, got = [[a(torch.zeros(1, device="cuda")), a(torch.full((rows, cols), 7.0, device="cuda"))] for _ in range(2)]
    G.softmax_ce(a(x), a(lab), want[0], st)
    G.softmax_ce_grad(a(x), a(lab), g, want[1], st)
    assert G.softmax_ce_both(a(x), a(lab), g, *got, st)
    assert torch.equal(want[0].t, got[0].t) and torch.equal(want[1].t, got[1].t)
    if G.softmax_ce_smooth(a(x), a(ids), 0.9, 1e-4, want[0], st):
        assert G.softmax_ce_grad_smooth(a(x), a(ids), 0.9, 1e-4, g, want[1], st)
        assert G.softmax_ce_both_smooth(a(x), a(ids), 0.9, 1e-4, g, *got, st)
        assert torch.equal(want[0].t, got[0].t) and torch.equal(want[1].t, got[1].t)
    else:
        assert not G.softmax_ce_both_smooth(a(x), a(ids), 0.9, 1e-4, g, *got, st)
