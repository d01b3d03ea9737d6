"""A residual addition with its ReLU computed by the batch norm before it, and the sum of two gradients by the later
convolution: the plan on the host, the kernels on the GPU."""
import numpy as np
import pytest
import torch

import test_step_plan as base
from tsplit_b200 import gpu_ops as ad, ndarray
from tsplit_b200.executors import step_plan
from tsplit_b200.models import resnet
from tsplit_b200.ops import _gpu as G
from tsplit_b200.ops.conv import Conv2dGradDataOp
from tsplit_b200.ops.norm import BatchNormOp, np_bn_forward


@pytest.mark.parametrize("taken", [True, False])
def test_resnet(monkeypatch, taken):
    joins = []

    def forward_add(self, node, iv, add, out, stream):
        joins.append(node)
        if taken:
            x, scale, bias, add = (v.numpy_view() for v in list(iv) + [add])
            out.numpy_view()[...] = np.maximum(self.np_compute(node, [x, scale, bias]) + add, 0)
        return taken
    monkeypatch.setattr(BatchNormOp, "forward_add", forward_add)
    added = []

    def add_to(self, node, iv, out, stream):
        added.append(node)
        if taken:
            out.numpy_view()[...] += self.np_compute(node, [v.numpy_view() for v in iv])
        return taken
    monkeypatch.setattr(Conv2dGradDataOp, "add_to", add_to)
    plan = base._compare(monkeypatch, lambda: base._model(resnet(26, num_classes=10, image=32, width_div=8), 2), steps=2)
    assert len(joins) == 16
    # eight blocks; in three of them the input's two gradients, one of stride 2
    assert sorted(type(b.op).name for b in plan.joined.values()) == ["BatchNorm"] * 8 + ["Conv2dGradData"] * 3
    assert len(added) == 6 and all(n.inputs.count(b) == 1 for n, b in plan.joined.items())


def test_what_stays(monkeypatch):
    """A batch norm that is kept, read twice, or added to itself."""
    def build():
        x, s, b = (ad.Variable(n) for n in ("x", "s", "b"))
        norms = [ad.batch_normalization_op(x, s, b) for _ in range(3)]
        r = np.random.default_rng(0)
        return ([norms[0], ad.add_relu_op(x, norms[0]), ad.add_relu_op(norms[1], x), norms[1] + x, ad.add_relu_op(norms[2], norms[2])],
                {x: r.standard_normal((2, 4, 6, 6), np.float32), s: np.ones((1, 4, 1, 1), np.float32),
                 b: np.zeros((1, 4, 1, 1), np.float32)})
    assert not base._compare(monkeypatch, build).joined


def test_planning_searches_no_list_of_additions(monkeypatch):
    """Counted in comparisons of nodes, which do not depend on the machine."""
    def comparisons(inputs):
        w, xs, count = ad.Variable("w"), [ad.Variable("x%d" % i) for i in range(inputs)], [0]
        sums = [ad.conv2d_op(x, w, padding=1, stride=2) + ad.conv2d_op(x, w, padding=1, stride=2) for x in xs]
        nodes = [g for s, x in zip(sums, xs) for g in ad.gradients(ad.reduce_sum_op(s, [0, 1, 2, 3]), [x])]
        shapes = {x: (1, 2, 8, 8) for x in xs}
        shapes[w] = (2, 2, 3, 3)
        ex = ad.Executor(nodes, ctx=ndarray.cpu(0))
        ex.infer_shape(shapes)
        ex.memory_plan(shapes)
        with monkeypatch.context() as m:
            m.setattr(type(w), "__eq__", lambda a, b: (count.__setitem__(0, count[0] + 1), a is b)[1], raising=False)
            plan = step_plan.StepPlan(ex, set(shapes))
        assert len(plan.joined) == inputs
        return count[0]
    assert comparisons(80) <= 4 * comparisons(20) + 100


# one row, part of a tile, a last tile of one thread's half, channels of no power of two; column sums of its own
@pytest.mark.gpu
@pytest.mark.parametrize("n,c,h,w", [(1, 4, 1, 1), (2, 36, 5, 7), (1, 2052, 1, 2), (4, 64, 31, 33)])
def test_bits_of_separate_operators(n, c, h, w):
    ctx, eps = ndarray.gpu(0), 0.01

    def arr(shape, seed=0):
        a = ndarray.empty(shape, ctx, use_pool=False)
        a.t.copy_(torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda"))
        return a
    from tsplit_b200.stream import current_stream
    stream = current_stream(ctx)
    x, add, scale, bias = arr((n, c, h, w), 1), arr((n, c, h, w), 2), arr((1, c, 1, 1), 3), arr((1, c, 1, 1), 4)
    results = []
    for joint in (False, True):
        y, z = arr((n, c, h, w)), arr((n, c, h, w))
        stats = [arr((c,), 5) for _ in range(4)]
        if joint:
            assert G.bn_forward_add(None, 0, x, scale, bias, add, z, *stats, 0.9, eps, stream)
        else:
            G.bn_forward(x, scale, bias, y, *stats, 0.9, eps, False, stream)
            G.binary(G.BIN_ADD_RELU, y, add, z, stream)
        results.append([z.t.clone()] + [s.t.clone() for s in stats])
    for a, b in zip(*results):
        assert torch.equal(a, b)
    want = np.maximum(np_bn_forward(*(v.t.cpu().numpy() for v in (x, scale, bias)), eps)[0] + add.t.cpu().numpy(), 0)
    # a handful of roundings of values of this size
    np.testing.assert_allclose(results[1][0].cpu().numpy(), want, rtol=0, atol=2 ** -19 * max(np.abs(want).max(), 1.0))
