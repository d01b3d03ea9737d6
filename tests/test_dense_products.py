"""Bias and ReLU stored by the product's own launch: the plan on the host, the kernels on the GPU against separate operators."""
import numpy as np
import pytest
import torch

import test_step_plan as base
from tsplit_b200 import gpu_ops as ad, ndarray, optimizer
from tsplit_b200.models import mlp, transformer
from tsplit_b200.ops import _gpu as G


def _dense(calls, takes_relu, takes_bias=True):
    def run(products, ta, tb, stream):
        calls.append([(p[6] is not None, p[7] is not None) for p in products])
        if any(p[7] is not None for p in products) and not takes_relu or not takes_bias:
            return False
        for a, b, c, m, n, k, bias, relu in products:
            x, y = a.numpy_view(), b.numpy_view()
            c.numpy_view()[...] = np.matmul(x.T if ta else x, y.T if tb else y) + (0 if bias is None else bias.numpy_view())
            if relu is not None:
                relu.numpy_view()[...] = np.maximum(c.numpy_view(), 0)
        return True
    return run


@pytest.mark.parametrize("takes_relu,takes_bias", [(True, True), (False, True), (False, False)])
@pytest.mark.parametrize("name", ["transformer", "mlp"])
def test_models(monkeypatch, name, takes_relu, takes_bias):
    def build():
        if name == "transformer":
            t = transformer(vocab_size=40, d_model=16, num_heads=2, d_ff=32, num_blocks=1, maxlen1=6, maxlen2=7, batch_size=3)
            return [t.loss, t.logits] + ad.gradients(t.loss, t.variables), t.synthetic_batch()
        return base._model(mlp((20, 12, 8, 4)), 4)
    calls = []
    monkeypatch.setattr(G, "gemm_dense", _dense(calls, takes_relu, takes_bias))
    plan = base._compare(monkeypatch, build, steps=2)
    if name == "transformer":                # q, k, v and output of three attentions, two layers of two feed-forward blocks
        assert sum(1 for b, _ in plan.dense.values() if b is not None) == 16
        assert sum(1 for _, r in plan.dense.values() if r is not None) == 2
        if takes_bias:                       # what is refused once is not tried again
            assert sum(b for c in calls for b, _ in c) == 16 * 2 + (0 if takes_relu else 2)
    else:
        assert [v[0] for v in plan.dense.values()] == [None, None] and len(calls) == (4 if takes_relu else 2)


def test_what_is_not_a_bias(monkeypatch):
    """A product that is kept, or read twice, or whose row is computed, or two ReLUs: left as they are."""
    def build():
        x, w, b = (ad.Variable(n) for n in ("x", "w", "b"))
        m1 = ad.matmul_op(x, w)
        kept = m1 + ad.broadcasttoTF_op(b, m1)
        m2 = ad.matmul_op(x, w)
        row = ad.mul_byconst_op(b, 2.0)
        computed = m2 + ad.broadcasttoTF_op(row, m2)
        m3 = ad.matmul_op(x, w)
        twice = m3 + ad.broadcasttoTF_op(b, m3)
        both = ad.relu_op(twice) + ad.relu_op(twice) + m3
        r = np.random.default_rng(0)
        return [m1, kept, computed, both], {x: r.standard_normal((8, 12), np.float32), w: r.standard_normal((12, 16), np.float32),
                                            b: r.standard_normal((16,), np.float32)}
    calls = []
    monkeypatch.setattr(G, "gemm_dense", _dense(calls, True))
    plan = base._compare(monkeypatch, build)
    assert not plan.dense and not calls


def test_what_stands_behind_an_update_is_not_stored_before_it(monkeypatch):
    """A bias that an update between the product and the addition changes, and a ReLU of a value behind an update; the
    products in front of one keep theirs."""
    r = np.random.default_rng(0)
    xv, wv, bv = (r.standard_normal(s).astype(np.float32) for s in ((4, 8), (8, 12), (12,)))
    made = []

    def build():
        x, w, b = ad.Variable("x"), ad.Variable("w"), ad.Variable("b", value=bv.copy())
        p, plain = ad.matmul_op(x, w), ad.matmul_op(x, w)
        q = ad.matmul_op(x, w)
        early = q + ad.broadcasttoTF_op(b, q)
        train = optimizer.SGDOptimizer(0.5).minimize(ad.reduce_sum_op(ad.mul_op(early, early), [0, 1]), [b])
        made[:] = [q]
        return [early, train, ad.relu_op(p + ad.broadcasttoTF_op(b, p)), ad.relu_op(plain), ad.relu_op(early)], {x: xv, w: wv}
    monkeypatch.setattr(G, "gemm_dense", _dense([], True))
    plan = base._compare(monkeypatch, build, steps=2)
    assert [(q, relu) for q, (bias, relu) in plan.dense.items()] == [(made[0], None)]


# one tile; a K that is split, by a cluster and by two kernels; rows of no whole 16 bytes; tiles of 64, 128 and 256 columns,
# one and several per block; CTA pairs, one tile and several each, ragged ones; a group of small products, one of wider ones
@pytest.mark.gpu
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("m,n,k,count", [(64, 32, 40, 1), (111, 512, 128, 1), (100, 10, 64, 1), (64, 256, 784, 1), (200, 128, 25088, 1),
                                         (19200, 64, 96, 1), (19200, 128, 96, 1), (2560, 1000, 96, 1), (8192, 512, 256, 1),
                                         (9000, 2052, 64, 1), (512, 2048, 4096, 1), (96, 128, 128, 3), (1024, 512, 128, 2)])
def test_bits_of_separate_operators(m, n, k, count, ta, tb):
    ctx = ndarray.gpu(0)

    def arr(*shape, seed=0):
        a = ndarray.empty(shape, ctx, use_pool=False)
        a.t.copy_(torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda"))
        return a
    from tsplit_b200.stream import current_stream
    st = current_stream(ctx)
    sets = []
    for i in range(count):
        a = arr(*((k, m) if ta else (m, k)), seed=i)
        b = arr(*((n, k) if tb else (k, n)), seed=10 + i)
        sets.append((a, b, arr(n, seed=20 + i), [arr(m, n, seed=30) for _ in range(4)]))
    products = [(a, b, o[0], m, n, k, bias, o[1]) for a, b, bias, o in sets]
    relu = G.gemm_dense(products, ta, tb, st)
    if not relu:
        assert all(torch.equal(o[0].t, o[2].t) for _, _, _, o in sets)              # refused: untouched
        if not G.gemm_dense([p[:7] + (None,) for p in products], ta, tb, st):
            assert n % 4
            return
    for a, b, bias, o in sets:
        G.gemm(a, b, o[2], ta, tb, st, m=m, n=n, k=k, lda=a.shape[1], ldb=b.shape[1], ldc=n)
        want = o[2].t + bias.t
        assert torch.equal(o[0].t, want)
        assert torch.equal(o[1].t, want.clamp(min=0) if relu else o[3].t)
