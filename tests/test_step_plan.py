"""The issue order of the keep-all executors on the GPU, interpreted on the host: programs of element-wise operators,
views and joint copies give what the node-by-node NumPy oracle gives, and nothing moves past an update."""
import ctypes

import numpy as np
import pytest

from tsplit_b200 import gpu_ops as ad, ndarray, optimizer
from tsplit_b200.executors import step_plan
from tsplit_b200.models import lstm, mlp, resnet, transformer
from tsplit_b200.ops import _gpu as G

_UN = {G.UN_COPY: lambda x, a: x, G.UN_RELU: lambda x, a: np.maximum(x, 0), G.UN_SIGMOID: lambda x, a: 1 / (1 + np.exp(-x)),
       G.UN_TANH: lambda x, a: np.tanh(x), G.UN_SQRT: lambda x, a: np.sqrt(x), G.UN_RSQRT: lambda x, a: 1 / np.sqrt(x),
       G.UN_NEG: lambda x, a: -x, G.UN_ADDC: lambda x, a: x + a, G.UN_MULC: lambda x, a: x * a, G.UN_CDIV: lambda x, a: a / x}
_BIN = {G.BIN_ADD: np.add, G.BIN_MUL: np.multiply, G.BIN_DIV: np.divide, G.BIN_SUB: np.subtract,
        G.BIN_RELU_GRAD: lambda x, g: np.where(x > 0, g, np.where(x == 0, 0.5 * g, 0)),
        G.BIN_ADD_RELU: lambda x, y: np.maximum(x + y, 0), G.BIN_RELU_GRAD_OUT: lambda y, g: np.where(y > 0, g, 0)}


def _at(address, n):
    return np.ctypeslib.as_array((ctypes.c_float * int(n)).from_address(address))


def _pointwise(inputs, kinds, code, alpha, outs, slots, n, cols, stream):
    assert len(inputs) <= step_plan.MAX_IN <= slots + step_plan.MAX_IN and len(outs) <= step_plan.MAX_INS
    assert slots <= step_plan.MAX_SLOTS and len(inputs) <= slots and n % 4 == 0
    value = [None] * slots
    for k, (p, kind) in enumerate(zip(inputs, kinds)):
        value[k] = _at(p, n).copy() if kind == step_plan.FULL else np.resize(_at(p, cols if kind == step_plan.ROW else 1), n)
    for k, out in enumerate(outs):
        op, a, b, dst = code[4 * k:4 * k + 4]
        if op == G.UN_FILL:
            v = np.full(n, alpha[k], np.float32)
        elif op < 32:
            v = _UN[op](value[a], np.float32(alpha[k])).astype(np.float32)
        else:
            v = _BIN[op - 32](value[a], value[b]).astype(np.float32)
        value[dst] = v
        if out:
            _at(out, n)[:] = v


class _HostPlan(step_plan.StepPlan):
    def _node(self, n, vals, stream):
        out = self.arrays.get(n)
        ins = [v.numpy_view() if isinstance(v, ndarray.NDArray) else v for v in (vals[i] for i in n.inputs)]
        n.op.compute(n, ins, out.numpy_view() if out is not None else None, True, None)
        vals[n] = out
        for key in ("dscale", "dbias"):
            if "np_" + key in getattr(n, "state", {}):
                n.state[key] = ndarray.array(n.state["np_" + key], ndarray.cpu(0))


def _smooth(grad, taken):
    """``softmax_ce_smooth`` / ``softmax_ce_grad_smooth`` in NumPy; ``taken``: False as for a shape it does not cover."""
    def run(logits, ids, on, off, *rest):
        if not taken:
            return False
        x, out = logits.numpy_view(), rest[1 if grad else 0].numpy_view()
        lab = np.where(np.arange(x.shape[1])[None, :] == ids.numpy_view().reshape(-1, 1), np.float32(on), np.float32(off))
        p = np.exp(x - x.max(1, keepdims=True))
        p /= p.sum(1, keepdims=True)
        out[...] = (p - lab) * rest[0].numpy_view() / x.shape[0] if grad else np.mean(-(lab * np.log(p)).sum(1))
        return True
    return run


def _gemm_group(products, ta, tb, stream):
    assert 2 <= len(products) <= step_plan.MAX_GROUP
    for a, b, c, m, n, k in products:
        x, y = a.numpy_view(), b.numpy_view()
        c.numpy_view()[...] = np.matmul(x.T if ta else x, y.T if tb else y)
        assert c.shape == (m, n) and k <= step_plan.GROUP_K
    return True


def _colsum_group(items, stream):
    assert 2 <= len(items) <= step_plan.MAX_GROUP
    for x, y in items:
        assert len(x.shape) == 2 and x.shape[0] <= step_plan.GROUP_ROWS
        y.numpy_view()[...] = x.numpy_view().sum(0).reshape(y.shape)
    return True


def _run(monkeypatch, nodes, feed, steps=1, taken=True):
    monkeypatch.setattr(G, "pointwise", _pointwise)
    monkeypatch.setattr(G, "gemm_group", _gemm_group if taken else lambda *a: False)
    monkeypatch.setattr(G, "colsum_group", _colsum_group if taken else lambda *a: False)
    monkeypatch.setattr(G, "softmax_ce_smooth", _smooth(False, taken))
    monkeypatch.setattr(G, "softmax_ce_grad_smooth", _smooth(True, taken))
    monkeypatch.setattr(G, "multi_copy", lambda s, d, st: [x.numpy_view().__setitem__(Ellipsis, y.numpy_view()) for x, y in zip(d, s)])
    ex = ad.Executor(nodes, ctx=ndarray.cpu(0))
    fed = {k: ndarray.array(v, ndarray.cpu(0)) for k, v in feed.items()}
    shapes = {k: v.shape for k, v in fed.items()}
    ex.infer_shape(shapes)
    ex.memory_plan(shapes)
    plan = _HostPlan(ex, set(fed))
    for _ in range(steps):
        vals = dict(fed)
        plan.run(ex, vals)
    return plan, [np.array(vals[n].numpy_view()) if isinstance(vals[n], ndarray.NDArray) else vals[n] for n in nodes]


def _compare(monkeypatch, build, steps=1, least=0, taken=True):
    nodes, feed = build()
    ex = ad.Executor(nodes)
    for _ in range(steps):
        want = ex.run(feed)
    nodes, feed = build()
    plan, got = _run(monkeypatch, nodes, feed, steps, taken)
    assert sum(1 for a in plan.actions if a[0] == "program") >= least
    for w, g in zip(want, got):
        if w is not None:
            # the oracle and the interpreter round alike, but for the order in which gradients meet
            np.testing.assert_allclose(g, w, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(w).max())))
    return plan


def _model(m, batch):
    x, y = m.synthetic_batch(batch)
    opt = optimizer.SGDOptimizer(0.1)
    train = opt.minimize(m.loss)
    return [m.loss, m.y, train] + m.variables, {m.X: x, m.y_: y}


@pytest.mark.parametrize("name,least", [("lstm", 6), ("mlp", 0), ("resnet", 1), ("transformer", 2)])
def test_models(monkeypatch, name, least):
    def build():
        if name == "transformer":
            t = transformer(vocab_size=40, d_model=16, num_heads=2, d_ff=32, num_blocks=1, maxlen1=6, maxlen2=7, batch_size=3)
            return [t.loss, t.logits] + ad.gradients(t.loss, t.variables), t.synthetic_batch()
        m = {"lstm": lambda: lstm(steps=4, features=8, hidden=12, num_classes=5), "mlp": lambda: mlp((20, 12, 8, 4)),
             "resnet": lambda: resnet(26, num_classes=4, image=32, width_div=16)}[name]()
        return _model(m, 4)
    plan = _compare(monkeypatch, build, steps=1, least=least)
    assert any(a[0] == "products" for a in plan.actions) or name not in ("lstm", "transformer")
    if name == "resnet":
        assert any(a[0] == "copies" and len(a[1]) > 10 for a in plan.actions)


@pytest.mark.parametrize("form", ["deep", "wide products", "wide sums", "one value, many readers"])
def test_planning_takes_time_in_proportion_to_the_graph(form):
    """The plan is made in the first pass over a feed shape; counted in calls, which do not depend on the machine."""
    import sys

    def calls(size):
        x, w, c = ad.Variable("x"), ad.Variable("w"), ad.Variable("c")
        shapes = {x: (8, 20), w: (20, 20), c: (20,)}
        if form == "deep":
            h = x
            for _ in range(size):
                h = ad.tanh_op(ad.matmul_op(h, w) + ad.broadcasttoTF_op(c, x))
            nodes = [h] + ad.gradients(ad.reduce_sum_op(h, [0, 1]), [w, c])
        elif form == "wide products":
            nodes = [ad.matmul_op(ad.mul_byconst_op(x, float(j)), w) for j in range(size)]
        elif form == "wide sums":
            nodes = [ad.reduce_sum_op(ad.mul_byconst_op(x, float(j)), [0]) for j in range(size)]
        else:
            s = ad.tanh_op(x)
            nodes = [ad.mul_op(s, ad.mul_byconst_op(x, float(j))) for j in range(size)]
        ex = ad.Executor(nodes, ctx=ndarray.cpu(0))
        ex.infer_shape(shapes)
        ex.memory_plan(shapes)
        count = [0]

        def profile(frame, event, arg):
            count[0] += event in ("call", "c_call")
        sys.setprofile(profile)
        try:
            step_plan.StepPlan(ex, set(shapes))
        finally:
            sys.setprofile(None)
        return count[0], len(ex.topo_order)
    (few, n), (many, n4) = calls(100), calls(400)
    assert many <= 1.15 * few * n4 / n and many <= 90 * n4


def _arrays(*shapes):
    r = np.random.RandomState(0)
    return [r.standard_normal(s).astype(np.float32) for s in shapes]


@pytest.mark.parametrize("shape", [(4, 8), (3, 5), (2, 3, 4), (1, 1), (2, 4, 3, 2)])
def test_forms_of_operands(monkeypatch, shape):
    """Whole operands, a row, a number first and second, the same operand twice, results that are kept, read by a
    reduction in the middle of a chain, and read through reshapes; sizes that are no multiple of four run node by node."""
    xv, zv, bv, sv = _arrays(shape, shape, shape[-1:], (1,))

    def build():
        x, z, b = (ad.Variable(k) for k in "xzb")
        s = ad.Variable("s", value=sv, trainable=False)
        a = ad.relu_op(x + ad.broadcasttoTF_op(b, x))
        c = ad.mul_op(a, a) + z
        kept = ad.sigmoid_op(c)
        total = ad.reduce_sum_op(kept, list(range(len(shape))))         # (1,): read back as a number
        by_number = ad.mul_op(total, ad.tanh_op(c)) + ad.mul_op(kept, s)
        flat = ad.array_reshape_op(ad.tanh_op(c), (-1,))
        e = ad.array_reshape_op(ad.mul_byconst_op(flat, 0.5), shape) + kept
        out = ad.array_reshape_op(e, (-1, 1))
        grads = ad.gradients(ad.reduce_sum_op(ad.mul_op(out, out), [0, 1]), [x, z, b])
        return [kept, out, flat, e, by_number] + grads, {x: xv, z: zv, b: bv, s: sv}
    _compare(monkeypatch, build)


def test_long_chains_are_cut(monkeypatch):
    """More operators, inputs and live values than one program holds."""
    vals = _arrays(*[(8, 4)] * 40)

    def build():
        xs = [ad.Variable("x%d" % i) for i in range(40)]
        ys = [ad.tanh_op(x) for x in xs]
        acc = ys[0]
        for i in range(1, 40):
            acc = ad.add_op(ad.mul_op(acc, ys[i]), ys[(7 * i) % 40])
        return [acc], dict(zip(xs, vals))
    _compare(monkeypatch, build, least=2)


def test_order_around_an_update(monkeypatch):
    """Values computed from a parameter before its update and after it, over three steps."""
    wv, xv = _arrays((8, 4), (2, 8))

    def build():
        x, w = ad.Variable("x"), ad.Variable("w", value=wv.copy())
        before = ad.mul_byconst_op(w, 2.0)
        y = ad.matmul_op(x, ad.relu_op(w))
        loss = ad.reduce_sum_op(ad.mul_op(y, y), [0, 1])
        train = optimizer.SGDOptimizer(0.05).minimize(loss)
        after = ad.addbyconst_op(ad.mul_byconst_op(w, 3.0), 1.0)
        return [loss, before, train, after], {x: xv}
    _compare(monkeypatch, build, steps=3)


def test_a_feed_in_another_layout_runs_node_by_node(monkeypatch):
    xv, zv = _arrays((4, 8), (4, 8))
    x, z = ad.Variable("x"), ad.Variable("z")
    out = ad.relu_op(ad.mul_op(x, z))
    plan, got = _run(monkeypatch, [out], {x: xv, z: zv})
    assert [a[0] for a in plan.actions] == ["program"]
    import torch
    vals = {x: ndarray.from_tensor(torch.from_numpy(np.ascontiguousarray(xv.T)).t(), ndarray.cpu(0)),
            z: ndarray.array(zv, ndarray.cpu(0))}
    plan.run(type("E", (), {"stream": None})(), vals)
    np.testing.assert_array_equal(vals[out].numpy_view(), got[0])


@pytest.mark.parametrize("taken", [True, False])
def test_constants_are_read_in_every_step(monkeypatch, taken):
    """An operator's number (``const_attr``) may change between steps; label smoothing is made of such operators, too."""
    xv, yv = _arrays((6, 12), (6, 12))
    x, y, i = (ad.Variable(k) for k in "xyi")
    scaled = ad.mul_byconst_op(x, 2.0)
    shifted = ad.addbyconst_op(scaled, 1.0)
    over = ad.div_const_op(3.0, ad.addbyconst_op(ad.mul_op(shifted, shifted), 0.5))
    rate = ad.mul_byconst_op(ad.one_hot_op(i, 12), 0.9)
    floor = ad.addbyconst_op(rate, 0.1 / 12)
    loss = ad.softmaxcrossentropy_op(y, floor)
    nodes = [over, loss] + ad.gradients(loss, [y])
    feed = {x: xv, y: yv, i: np.array([0, 3, 11, 5, 5, 2], np.float32)}
    plan, first = _run(monkeypatch, nodes, feed, taken=taken)
    assert {"program", "smooth"} <= {a[0] for a in plan.actions}
    scaled.const_attr, shifted.const_attr, over.const_attr, rate.const_attr, floor.const_attr = -1.5, 0.25, 7.0, 0.6, 0.4 / 12
    vals = {k: ndarray.array(v, ndarray.cpu(0)) for k, v in feed.items()}
    plan.run(type("E", (), {"stream": None})(), vals)
    want = ad.Executor(nodes).run(feed)
    for n, w, f in zip(nodes, want, first):
        assert not np.allclose(f, w, rtol=1e-3)
        np.testing.assert_allclose(vals[n].numpy_view(), w, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("taken", [True, False])
def test_products_that_are_ready_together(monkeypatch, taken):
    """Products of all four transpositions, too long and too wide ones, one that reads another, more than one launch."""
    xv, wv, longv, widev = _arrays((6, 20), (20, 6), (20, 600), (600, 3000))

    def build():
        x, w, l, b = (ad.Variable(k) for k in "xwlb")
        outs = [ad.matmul_op(x, w), ad.matmul_op(w, x, True, True), ad.matmul_op(x, x, True), ad.matmul_op(x, x, False, True)]
        outs += [ad.matmul_op(ad.mul_byconst_op(x, float(j)), w) for j in range(40)]
        outs += [ad.matmul_op(outs[0], outs[5]), ad.matmul_op(ad.matmul_op(x, l), b), ad.matmul_op(x, l)]
        return outs, {x: xv, w: wv, l: longv, b: widev}
    plan = _compare(monkeypatch, build, taken=taken)
    groups = [a[1] for a in plan.actions if a[0] == "products"]
    assert sum(len(g) for g in groups) >= 40 and max(len(g) for g in groups) == step_plan.MAX_GROUP


def test_a_product_that_no_group_takes_leaves_the_others_together(monkeypatch):
    """Rows of 10 classes have to be padded, so that product runs by itself, not all that are ready with it."""
    xv, wv, cv = _arrays((6, 20), (20, 8), (20, 10))
    groups, alone, taken = [], [], _gemm_group
    node = _HostPlan._node

    def group(products, ta, tb, stream):
        if any(a.shape[1] % 4 or b.shape[1] % 4 for a, b, *_ in products):
            return False                                       # as the native entry does, for all of them
        groups.append(len(products))
        return taken(products, ta, tb, stream)
    monkeypatch.setitem(globals(), "_gemm_group", group)
    monkeypatch.setattr(_HostPlan, "_node", lambda self, n, vals, stream: (alone.append(n.op.name), node(self, n, vals, stream)))

    def build():
        x, w, c = (ad.Variable(k) for k in "xwc")
        outs = [ad.matmul_op(ad.mul_byconst_op(x, float(j)), w) for j in range(5)]
        return outs + [ad.matmul_op(x, c)], {x: xv, w: wv, c: cv}
    plan = _compare(monkeypatch, build)
    assert [len(a[1]) for a in plan.actions if a[0] == "products"] == [6]
    assert groups == [5] and alone.count("MatMul") == 1


@pytest.mark.parametrize("taken", [True, False])
def test_sums_that_are_ready_together(monkeypatch, taken):
    """Column sums with and without the reduced dimension kept, sums over other axes and over too many rows."""
    xv, yv, longv = _arrays((6, 20), (5, 6, 8), (600, 4))

    def build():
        x, y, l = (ad.Variable(k) for k in "xyl")
        outs = [ad.reduce_sum_op(ad.mul_byconst_op(x, float(j + 1)), [0]) for j in range(20)]
        outs += [ad.reduce_sum_op(x, [0], True), ad.reduce_sum_op(x, [1]), ad.reduce_sum_op(x, [0, 1]),
                 ad.reduce_sum_op(y, [0, 1]), ad.reduce_sum_op(l, [0])]
        return outs, {x: xv, y: yv, l: longv}
    plan = _compare(monkeypatch, build, taken=taken)
    assert [len(a[1]) for a in plan.actions if a[0] == "sums"] == [16, 5]


@pytest.mark.parametrize("form", ["plain", "smooth", "shifted twice", "kept", "read elsewhere", "two losses", "fed"])
@pytest.mark.parametrize("taken", [True, False])
def test_labels_from_ids(monkeypatch, form, taken):
    """One-hot labels that only cross-entropies read are not made; all others are."""
    xv, yv = _arrays((6, 12), (6, 12))
    ids = np.array([[0, 3, 11], [5, 5, 2]], np.float32)

    def build():
        x, y, i = (ad.Variable(k) for k in "xyi")
        lab = ad.array_reshape_op(ad.one_hot_op(i, 12), (-1, 12))
        if form != "plain":
            lab = ad.addbyconst_op(ad.mul_byconst_op(lab, 0.9), 0.1 / 12)
        if form == "shifted twice":
            lab = ad.mul_byconst_op(ad.addbyconst_op(lab, 0.25), 0.5)
        loss = ad.softmaxcrossentropy_op(x, lab)
        nodes = [loss] + ad.gradients(loss, [x])
        feed = {x: xv, i: ids}
        if form == "kept":
            nodes.append(lab)
        if form == "read elsewhere":
            nodes.append(ad.reduce_sum_op(lab, [0]))
        if form == "two losses":
            feed[y] = yv
            nodes.append(ad.softmaxcrossentropy_op(y, lab))
        if form == "fed":
            feed[lab] = np.abs(yv)
        return nodes, feed
    plan = _compare(monkeypatch, build, taken=taken)
    made = form in ("kept", "read elsewhere", "fed")
    assert sum(1 for a in plan.actions if a[0] == "smooth") == (0 if made else 3 if form == "two losses" else 2)


def test_labels_that_are_refused_are_made_once_a_step(monkeypatch):
    """The loss and its gradient both ask for labels from ids; a class count that the kernels do not cover costs the four
    operators of the label chain, not eight."""
    xv, = _arrays((6, 12))
    x, i = ad.Variable("x"), ad.Variable("i")
    lab = ad.addbyconst_op(ad.mul_byconst_op(ad.array_reshape_op(ad.one_hot_op(i, 12), (-1, 12)), 0.9), 0.1 / 12)
    loss = ad.softmaxcrossentropy_op(x, lab)
    nodes = [loss] + ad.gradients(loss, [x])
    feed = {x: xv, i: np.array([[0, 3, 11], [5, 5, 2]], np.float32)}
    ran = []
    node = _HostPlan._node
    monkeypatch.setattr(_HostPlan, "_node", lambda self, n, vals, stream: (ran.append(n.op.name), node(self, n, vals, stream)))
    plan, got = _run(monkeypatch, nodes, feed, steps=2, taken=False)
    assert [ran.count(k) for k in ("OneHot", "Reshape", "MulConst", "AddConst")] == [2, 2, 2, 2]        # of two steps
    for w, g in zip(ad.Executor(nodes).run(feed), got):
        np.testing.assert_allclose(g, w, rtol=1e-5, atol=1e-6)


def test_labels_are_older_than_an_update_of_their_ids(monkeypatch):
    """A cross-entropy behind the update reads the labels that were made in front of it."""
    xv, = _arrays((6, 12))
    old, new = np.array([0, 3, 11, 5, 5, 2], np.float32), np.array([1, 2, 3, 4, 5, 6], np.float32)

    def build():
        x, t, i = ad.Variable("x"), ad.Variable("t"), ad.Variable("i", value=old.copy())
        lab = ad.addbyconst_op(ad.mul_byconst_op(ad.one_hot_op(i, 12), 0.9), 0.01)
        early = ad.softmaxcrossentropy_op(x, lab)
        diff = i + ad.opposite_op(t)
        train = optimizer.SGDOptimizer(0.5).minimize(ad.reduce_sum_op(ad.mul_op(diff, diff), [0]), [i])     # i = t
        return [early, train, ad.softmaxcrossentropy_op(ad.mul_byconst_op(x, 2.0), lab)], {x: xv, t: new}
    assert not _compare(monkeypatch, build).smooth


# one group of four; a row length that is no power of two; the last size of the short blocks and the first of the long
# ones; a tensor past the limit for many values
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 4), (3, 20), (64 * 148, 4), (64 * 148 + 1, 4), (2049, 4096)])
def test_programs_give_the_bits_of_the_single_kernels(shape):
    import torch
    ctx = ndarray.gpu(0)
    xv, zv, bv = _arrays(shape, shape, shape[-1:])
    x, z, b = (ad.Variable(k) for k in "xzb")
    s = ad.Variable("s", value=np.full((1,), 0.75, np.float32), trainable=False)
    a = ad.relu_op(x + ad.broadcasttoTF_op(b, x))
    c = ad.sigmoid_op(ad.mul_op(a, z)) + ad.tanh_op(ad.div_op(z, ad.addbyconst_op(ad.mul_op(x, x), 1.0)))
    d = ad.add_relu_op(ad.opposite_op(c), ad.mul_op(ad.sqrt_op(ad.mul_op(z, z)), s))
    e = ad.relu_gradient_op(d, ad.div_const_op(2.0, ad.addbyconst_op(a, 1.5)))
    f = ad.relu_out_gradient_op(a, ad.mul_byconst_op(e, 0.3)) + ad.array_reshape_op(ad.array_reshape_op(d, (-1,)), shape)
    nodes = [a, c, f, ad.rsqrt_op(ad.addbyconst_op(ad.mul_op(f, f), 0.5))]
    ex = ad.Executor(nodes, ctx=ctx)
    feed = {k: ndarray.array(v, ctx, use_pool=False) for k, v in ((x, xv), (z, zv), (b, bv))}
    got = [o.t.clone() for o in ex.run(feed)]
    plan = ex._step_plan
    assert any(k == "program" for k, _ in plan.actions)
    vals = dict(feed)
    vals[s] = s.tensor_value
    for kind, what in plan.actions:
        for n in what.members if kind == "program" else [what]:
            if kind == "view":
                vals[n] = plan.arrays[n]
            else:
                plan.arrays[n].t.fill_(-1.0)
                plan._node(n, vals, ex.stream)
    ex.stream.sync()
    for n, g in zip(nodes, got):
        assert torch.equal(vals[n].t, g), n.desc


@pytest.mark.gpu
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_product_groups_give_the_bits_of_single_products(ta, tb):
    import torch
    from tsplit_b200.stream import current_stream
    ctx, st = ndarray.gpu(0), current_stream(ndarray.gpu(0))
    r = torch.Generator(device="cuda").manual_seed(2)
    # one element, ragged tiles, several tiles, the longest sum that is not split; then a group with wider tiles
    for sizes in ([(4, 4, 4), (128, 128, 128), (130, 68, 28), (300, 200, 480), (1, 132, 64)], [(256, 1000, 96)] * 8,
                  [(64, 64, 32)] * 16, [(128, 256, 40), (8, 12, 36)]):
        items, single = [], []
        for m, n, k in sizes:
            m4, n4 = (m + 3) // 4 * 4 if ta else m, n if tb else (n + 3) // 4 * 4
            a = torch.randn((k, m4) if ta else (m4, k), generator=r, device="cuda")
            b = torch.randn((n4, k) if tb else (k, n4), generator=r, device="cuda")
            c, d = (torch.full((m4, n4), 5.0, device="cuda") for _ in range(2))
            items.append(tuple(ndarray.from_tensor(t, ctx) for t in (a, b, c)) + (m4, n4, k))
            G.gemm(items[-1][0], items[-1][1], ndarray.from_tensor(d, ctx), ta, tb, st, m=m4, n=n4, k=k, lda=a.shape[1],
                   ldb=b.shape[1], ldc=n4)
            single.append(d)
        assert G.gemm_group(items, ta, tb, st)
        for it, d in zip(items, single):
            assert torch.equal(it[2].t, d)
    a = ndarray.from_tensor(torch.zeros((2048, 2048), device="cuda"), ctx)
    assert not G.gemm_group([(a, a, a, 2048, 2048, 2048)], ta, tb, st)           # no small product: refused, untouched


@pytest.mark.gpu
def test_operators_are_timed_after_a_planned_step():
    t = transformer(vocab_size=512, d_model=16, num_heads=2, d_ff=32, num_blocks=1, maxlen1=8, maxlen2=9, batch_size=4)
    ex = ad.recomputeExecutor([t.loss] + ad.gradients(t.loss, t.variables), ctx=ndarray.gpu(0), policy="speed")
    feed = t.synthetic_batch()
    table = ex.measure_ops(feed, repeats=1)
    names = {n.op.name for n in table}
    assert {"OneHot", "Reshape", "MulConst", "SoftmaxCrossEntropy", "MatMul"} <= names and min(table.values()) > 0
