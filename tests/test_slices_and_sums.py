"""Slices that products read in place, and column sums that wait for a launch of their own size."""
import numpy as np
import pytest
import torch

import test_step_plan as base
from tsplit_b200 import gpu_ops as ad, ndarray, optimizer
from tsplit_b200.executors import step_plan
from tsplit_b200.models import lstm
from tsplit_b200.ops import _gpu as G


def _dense(products, ta, tb, stream):
    for a, b, c, m, n, k, bias, relu in products:
        x, y = a.numpy_view(), b.numpy_view()
        c.numpy_view()[...] = np.matmul(x.T if ta else x, y.T if tb else y) + (0 if bias is None else bias.numpy_view())
        if relu is not None:
            relu.numpy_view()[...] = np.maximum(c.numpy_view(), 0)
    return True


@pytest.mark.parametrize("features,taken", [(8, True), (8, False), (7, True)])
def test_recurrent_steps(monkeypatch, features, taken):
    """Rows of the fed batch are sliced for every step: read in place, or copied where they do not begin on 16 bytes."""
    copies = []

    def compute(self, node, ins, out, *rest):
        copies.append(node)
        out = out.numpy_view() if isinstance(out, ndarray.NDArray) else out
        x = ins[0].numpy_view() if isinstance(ins[0], ndarray.NDArray) else ins[0]
        out[...] = self.np_compute(node, [x])
    monkeypatch.setattr(step_plan.SliceOp, "compute", compute)
    monkeypatch.setattr(G, "gemm_dense", _dense if taken else lambda *a: False)
    plan = base._compare(monkeypatch, lambda: base._model(lstm(steps=6, features=features, hidden=12, num_classes=5), 4), taken=taken)
    assert len(plan.sliced) == 6 and sum(1 for a in plan.actions if a[0] == "slice") == 6
    assert len(plan.sliced.intersection(copies)) == (6 if features % 4 else 0)
    groups = [len(a[1]) for a in plan.actions if a[0] == "sums"]
    assert sum(groups) >= 20 and max(groups) == step_plan.MAX_GROUP and len(groups) <= 3


def test_which_slices_are_copied(monkeypatch):
    """One that is kept, one that something else reads, one of a computed value."""
    def build():
        x, w = ad.Variable("x"), ad.Variable("w")
        kept, read, in_place = (ad.slice_op(x, (0, 4 * i), (-1, 4)) for i in range(3))
        inner = ad.slice_op(ad.mul_byconst_op(x, 2.0), (2, 0), (4, 4))
        r = np.random.default_rng(0)
        return ([kept, ad.matmul_op(kept, w), ad.matmul_op(read, w), read * 3.0, ad.matmul_op(in_place, w), ad.matmul_op(inner, w)],
                {x: r.standard_normal((8, 12), np.float32), w: r.standard_normal((4, 12), np.float32)})
    monkeypatch.setattr(G, "gemm_dense", _dense)
    assert len(base._compare(monkeypatch, build).sliced) == 1


@pytest.mark.parametrize("steps", [1, 2])
def test_a_slice_is_older_than_the_update_behind_it(monkeypatch, steps):
    """A product behind the update reads what was sliced before it; slices that are read on one side only stay in place."""
    r = np.random.default_rng(0)
    xv, zv, wv = (r.standard_normal(s).astype(np.float32) for s in ((4, 8), (4, 8), (8, 12)))
    made = []

    def compute(self, node, ins, out, *rest):
        out, x = (v.numpy_view() if isinstance(v, ndarray.NDArray) else v for v in (out, ins[0]))
        out[...] = self.np_compute(node, [x])
    monkeypatch.setattr(step_plan.SliceOp, "compute", compute)
    monkeypatch.setattr(G, "gemm_dense", _dense)

    def build():
        x, z, w = ad.Variable("x"), ad.Variable("z"), ad.Variable("w", value=wv.copy())
        both, early = ad.slice_op(w, (0, 4), (8, 4)), ad.slice_op(w, (0, 0), (8, 4))
        h = ad.matmul_op(x, both) + ad.matmul_op(x, early)
        train = optimizer.SGDOptimizer(0.05).minimize(ad.reduce_sum_op(ad.mul_op(h, h), [0, 1]), [w])
        late = ad.slice_op(w, (0, 8), (8, 4))
        made[:] = [both, early, late]
        return [h, train, ad.matmul_op(z, both), ad.matmul_op(z, late)], {x: xv, z: zv}
    plan = base._compare(monkeypatch, build, steps=steps)
    assert plan.sliced == set(made[1:])


@pytest.mark.gpu
@pytest.mark.parametrize("steps,features,batch", [(3, 28, 64), (4, 6, 5), (3, 4, 1)])
def test_step_on_the_gpu(monkeypatch, steps, features, batch):
    """Gradients with every slice read in place, with launches that refuse (products alone, which read whole arrays), and
    with every slice copied."""
    ctx = ndarray.gpu(0)
    outs = []
    for how in ("in place", "refused", "copied"):
        if how == "refused":
            monkeypatch.setattr(G, "gemm_group", lambda *a: False)
            monkeypatch.setattr(G, "gemm_dense", lambda *a: False)
        elif how == "copied":
            monkeypatch.undo()
            monkeypatch.setattr(step_plan.StepPlan, "_is_sliced", lambda self, n: False)
        m = lstm(steps=steps, features=features, hidden=32, num_classes=10)
        x, y = m.synthetic_batch(batch)
        ex = ad.Executor([m.loss] + ad.gradients(m.loss, list(m.variables)), ctx=ctx)
        feed = {m.X: ndarray.array(x, ctx), m.y_: ndarray.array(y, ctx)}
        outs.append([o.t.clone() for o in ex.run(feed)])
    for other in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(outs[0], other))


@pytest.mark.gpu
def test_operators_are_timed_after_a_step_with_slices_in_place():
    m = lstm(steps=3, features=8, hidden=32, num_classes=12)
    x, y = m.synthetic_batch(16)
    ex = ad.recomputeExecutor([m.loss] + ad.gradients(m.loss, list(m.variables)), ctx=ndarray.gpu(0), policy="speed")
    table = ex.measure_ops({m.X: x, m.y_: y}, repeats=1)
    assert {"Slice", "MatMul"} <= {n.op.name for n in table} and min(table.values()) > 0
