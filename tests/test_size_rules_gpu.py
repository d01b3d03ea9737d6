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


@pytest.mark.parametrize("sizes", [[-1, 5, 0, 3000, -2048], [0, -7], [4, -3]])
def test_optimizer_leaves_tensors_of_no_elements_alone(sizes):
    """Sizes of zero and below are tensors with nothing to update, not an error."""
    import ctypes
    n = len(sizes)
    ps, gs = ([_rand(max(k, 8), seed=j + 100 * i) for j, k in enumerate(sizes)] for i in range(2))
    before = [p.clone() for p in ps]
    ptrs = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() for t in ts])
    rc = G.lib().tsb_optimizer_step(ctypes.c_int(0), ctypes.c_int(n), ptrs(ps), ptrs(gs), None, None,
                                    (ctypes.c_int64 * n)(*sizes), (ctypes.c_float * 8)(0.5), ctypes.c_void_p(None))
    torch.cuda.synchronize()
    assert rc == 0
    for k, p, g, p0 in zip(sizes, ps, gs, before):
        k = max(k, 0)
        torch.testing.assert_close(p[:k], p0[:k] - 0.5 * g[:k], rtol=0, atol=2e-6)        # (contracted or not)
        assert torch.equal(p[k:], p0[k:])


# launches whose tiles are narrowed: one tile, a ragged one, the last number of wide tiles that is halved and the first
# that is not, and a batch; every combination of transposed operands
@pytest.mark.parametrize("m,n,k,batch", [(64, 256, 96, 1), (130, 300, 70, 1), (5, 129, 40, 1), (128 * 74, 256, 32, 1),
                                         (128 * 74 + 4, 256, 32, 1), (36, 132, 64, 20)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_gemm_tiles_of_small_launches(m, n, k, batch, ta, tb):
    a, b = _rand(batch, k, m) if ta else _rand(batch, m, k), _rand(batch, n, k, seed=1) if tb else _rand(batch, k, n, seed=1)
    c = torch.full((batch, m, n), 9.0, device="cuda")
    ctx = ndarray.gpu(0)
    G.gemm(ndarray.from_tensor(a, ctx), ndarray.from_tensor(b, ctx), ndarray.from_tensor(c, ctx), ta, tb, _stream(),
           batch=batch, m=m, n=n, k=k, sa=m * k, sb=n * k, sc=m * n, lda=a.shape[2], ldb=b.shape[2], ldc=n)
    x, y = (a.transpose(1, 2) if ta else a).double(), (b.transpose(1, 2) if tb else b).double()
    # an operand cut to 10 mantissa bits is at most 2^-10 off, so a product is 2^-9 of its magnitude; fp32 sums add less
    assert torch.all((c.double() - x @ y).abs() <= 2.2e-3 * (x.abs() @ y.abs()) + 1e-6)


# the same for convolutions: 7 x 7 pixels of 512 channels (4 x 2 wide tiles), a ragged width, 37 and 38 tiles of a batch
@pytest.mark.parametrize("n,c,hw,o,k", [(8, 64, 7, 512, 3), (2, 32, 9, 200, 1), (37, 32, 11, 256, 1), (38, 32, 11, 256, 3)])
def test_convolution_tiles_of_small_launches(n, c, hw, o, k):
    x, w, dy = _rand(n, c, hw, hw), _rand(o, c, k, k, seed=1), _rand(n, o, hw, hw, seed=2)
    y, dx = _arr(torch.zeros(n, o, hw, hw, device="cuda")), _arr(torch.zeros(n, c, hw, hw, device="cuda"))
    conv = torch.nn.functional.conv2d
    grad = torch.nn.grad.conv2d_input
    part = ndarray.empty((2 * G.CONV_STAT_MAX_CHUNKS * o,), ndarray.gpu(0), use_pool=False)
    chunks = G.conv2d_fwd_stats(_arr(x), _arr(w), y, k // 2, k // 2, 1, part, _stream())
    xd, wd, dyd = x.double(), w.double(), dy.double()
    assert torch.all((y.t.double() - conv(xd, wd, padding=k // 2)).abs()
                     <= 2.2e-3 * conv(xd.abs(), wd.abs(), padding=k // 2) + 1e-6)
    G.conv2d(1, dx, _arr(w), _arr(dy), k // 2, k // 2, 1, _stream())
    assert torch.all((dx.t.double() - grad(x.shape, wd, dyd, padding=k // 2)).abs()
                     <= 2.2e-3 * grad(x.shape, wd.abs(), dyd.abs(), padding=k // 2) + 1e-6)
    if chunks:                         # the column sums are those of the rounded outputs, in fp32
        planes = part.t.view(2, G.CONV_STAT_MAX_CHUNKS, o)[:, :chunks].double().sum(1)
        ys = y.t.double()
        torch.testing.assert_close(planes[0], ys.sum((0, 2, 3)), rtol=0, atol=1e-5 * float(ys.abs().sum((0, 2, 3)).max()))
        torch.testing.assert_close(planes[1], ys.square().sum((0, 2, 3)), rtol=1e-5, atol=1e-5)


# the shortest long row, the last that is not staged, the first and the last that are and the first past them; fewer
# rows than blocks and more; an id outside the classes
@pytest.mark.parametrize("cols", [512, 8188, 8192, 32000, 51200, 51204])
@pytest.mark.parametrize("rows", [1, 700])
def test_cross_entropy_of_long_rows(rows, cols):
    ctx = ndarray.gpu(0)
    x = 3 * _rand(rows, cols)
    ids = torch.randint(0, cols, (rows,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).float()
    if rows > 1:
        ids[1], ids[2], ids[3] = cols, 0, cols - 1
    on, off = np.float32(0.9) + np.float32(0.1 / cols), np.float32(0.1 / cols)
    lab = torch.full((rows, cols), float(off), device="cuda")
    inside = ids < cols
    lab[inside, ids[inside].long()] = float(on)
    g = torch.full((1,), 0.5, device="cuda")
    dense, smooth = [[torch.zeros(1, device="cuda"), torch.zeros(rows, cols, device="cuda")] for _ in range(2)]
    a = lambda t: ndarray.from_tensor(t, ctx)
    G.softmax_ce(a(x), a(lab), a(dense[0]), _stream())
    G.softmax_ce_grad(a(x), a(lab), a(g), a(dense[1]), _stream())
    assert G.softmax_ce_smooth(a(x), a(ids), float(on), float(off), a(smooth[0]), _stream())
    assert G.softmax_ce_grad_smooth(a(x), a(ids), float(on), float(off), a(g), a(smooth[1]), _stream())
    assert torch.equal(dense[1], smooth[1])
    lp = torch.log_softmax(x.double(), 1)
    ref = -(lab.double() * lp).sum(1).mean().reshape(1)
    # fp32 sums of some 10^4 terms of one sign per row, and the fast exponential's 2^-21
    for loss in (dense[0], smooth[0]):
        torch.testing.assert_close(loss.double(), ref, rtol=2e-5, atol=1e-5)
    torch.testing.assert_close(dense[1].double(), (lp.exp() - lab.double()) * 0.5 / rows, rtol=1e-4, atol=1e-6 * 0.5 / rows)


# masked classes (the lowest float, a common mask value, minus infinity): two of them, half of them, all of one thread's, and
# the labelled one; the loss from ids is finite, infinite or NaN where the one from dense labels is
@pytest.mark.parametrize("masked", ["two", "half", "a thread's", "the label"])
@pytest.mark.parametrize("value", [float(np.finfo(np.float32).min), -1e9, float("-inf")])
@pytest.mark.parametrize("cols", [512, 8192, 32000])
def test_cross_entropy_with_masked_classes(cols, value, masked):
    ctx = ndarray.gpu(0)
    rows = 5
    ids = torch.tensor([0., 7., cols - 1, cols // 2, cols], device="cuda")             # the last one: no class
    x = 3 * _rand(rows, cols)
    if masked == "two":
        x[:, 3], x[:, cols - 3] = value, value
    elif masked == "half":
        x[:, 1::2] = value
    elif masked == "a thread's":
        x[:, 8:12] = value
        x[:, 8 + 4 * 256:12 + 4 * 256] = value
        x[:, 8 + 4 * 512::4 * 512] = value
    else:
        x[torch.arange(4), ids[:4].long()] = value
    a = lambda t: ndarray.from_tensor(t, ctx)
    g = torch.ones(1, device="cuda")
    for on, off in ((1.0, 0.0), (float(np.float32(0.9) + np.float32(0.1 / cols)), float(np.float32(0.1 / cols)))):
        lab = torch.full((rows, cols), off, device="cuda")
        lab[torch.arange(4), ids[:4].long()] = on
        for r in range(rows):                                                          # each row's loss by itself
            dense, smooth, row, i = torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda"), x[r:r + 1], ids[r:r + 1]
            G.softmax_ce(a(row), a(lab[r:r + 1]), a(dense), _stream())
            assert G.softmax_ce_smooth(a(row), a(i), on, off, a(smooth), _stream())
            lp = torch.log_softmax(row.double(), 1)
            want = -(lab[r:r + 1].double() * lp).sum().float()
            _stream().sync()
            for loss in (dense, smooth):               # fp32 sums of terms of one sign, as in the test above
                torch.testing.assert_close(loss[0], want, rtol=2e-5, atol=2e-5, equal_nan=True)
        dd, ds = torch.zeros(rows, cols, device="cuda"), torch.ones(rows, cols, device="cuda")
        G.softmax_ce_grad(a(x), a(lab), a(g), a(dd), _stream())
        assert G.softmax_ce_grad_smooth(a(x), a(ids), on, off, a(g), a(ds), _stream())
        _stream().sync()
        assert torch.equal(dd, ds)


@pytest.mark.parametrize("offset", [0.0, -37.0, 1000.0])
@pytest.mark.parametrize("cols", [512, 32000])
def test_cross_entropy_of_logits_with_a_common_offset(cols, offset):
    """The loss does not depend on what all logits of a row have in common, and its rounding hardly does."""
    ctx, rows = ndarray.gpu(0), 64
    x = _rand(rows, cols) + offset
    ids = torch.randint(0, cols, (rows,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(8)).float()
    a = lambda t: ndarray.from_tensor(t, ctx)
    on, off = float(np.float32(0.9) + np.float32(0.1 / cols)), float(np.float32(0.1 / cols))
    lab = torch.full((rows, cols), off, device="cuda")
    lab[torch.arange(rows), ids.long()] = on
    want = -(lab.double() * torch.log_softmax(x.double(), 1)).sum(1).mean()
    dense, smooth = torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda")
    G.softmax_ce(a(x), a(lab), a(dense), _stream())
    assert G.softmax_ce_smooth(a(x), a(ids), on, off, a(smooth), _stream())
    _stream().sync()
    # a logit of 1000 has a unit in the last place of 6e-5; its distance to the row's lse is rounded once, and rows average
    bound = 8 * 2.0 ** -24 * (float(want) + abs(offset) / 64 ** 0.5)
    assert abs(float(smooth[0]) - float(want)) <= bound and abs(float(dense[0]) - float(want)) <= bound


# outputs that leave by TMA store: ragged rows and columns of a block, one column block and many, batches, several
# splits; and those whose strides or sums do not allow it (a row of 130 + 1 floats, a base 4 bytes in, accumulation)
@pytest.mark.parametrize("m,n,k,batch,ldc,shift,accumulate", [
    (129, 68, 40, 1, 68, 0, False), (300, 260, 64, 3, 260, 0, False), (31, 12, 33, 5, 16, 0, False),
    (64, 256, 1024, 1, 256, 0, False), (512, 520, 96, 1, 640, 0, False), (130, 100, 64, 2, 131, 0, False),
    (130, 100, 64, 2, 132, 1, False), (130, 100, 64, 2, 132, 0, True), (1, 4, 4, 1, 4, 0, False)])
def test_gemm_output_forms(m, n, k, batch, ldc, shift, accumulate):
    ctx = ndarray.gpu(0)
    a, b = _rand(batch, m, k), _rand(batch, k, n, seed=1)
    room = torch.full((shift + batch * m * ldc + 8,), 2.0, device="cuda")
    c = room[shift:shift + batch * m * ldc].view(batch, m, ldc)
    G.gemm(ndarray.from_tensor(a, ctx), ndarray.from_tensor(b, ctx), ndarray.from_tensor(c, ctx), False, False, _stream(),
           batch=batch, m=m, n=n, k=k, sa=m * k, sb=n * k, sc=m * ldc, lda=k, ldb=n, ldc=ldc, accumulate=accumulate)
    x, y = a.double(), b.double()
    want = x @ y + (2.0 if accumulate else 0.0)
    assert torch.all((c[:, :, :n].double() - want).abs() <= 2.2e-3 * (x.abs() @ y.abs()) + 1e-6)
    assert torch.all(c[:, :, n:] == 2) and torch.all(room[:shift] == 2) and torch.all(room[shift + batch * m * ldc:] == 2)


# overlapping windows: tiles cut at both edges, one tile, windows that skip pixels, several channel blocks with a ragged
# one, padding as wide as the window allows, and windows too large for a tile's shared memory (two passes)
@pytest.mark.parametrize("n,c,h,w,k,pad,stride", [(2, 4, 17, 33, 3, 1, 2), (1, 36, 16, 16, 3, 1, 2), (1, 8, 15, 31, 3, 0, 2),
                                                  (2, 8, 20, 18, 3, 1, 1), (1, 8, 35, 20, 2, 0, 3), (1, 64, 9, 40, 5, 2, 2),
                                                  (1, 4, 24, 24, 9, 4, 1), (1, 4, 40, 40, 15, 7, 1), (3, 4, 1, 1, 1, 0, 1)])
def test_max_pool_gradient_tiles(n, c, h, w, k, pad, stride):
    x = torch.round(_rand(n, c, h, w) * 2) / 2                       # ties on purpose: the first maximum takes all
    ref_x = x.double().requires_grad_()
    ref_y = torch.nn.functional.max_pool2d(ref_x, k, stride, pad)
    dy = torch.round(_rand(*ref_y.shape, seed=1) * 8) / 8            # sums of eighths are exact
    y, dx = _arr(ref_y.detach().float()), _arr(torch.full_like(x, 7.0))
    G.pool_grad(0, _arr(x), y, _arr(dy), dx, k, k, pad, stride, _stream())
    # torch gives a tie to the last or first maximum depending on the layout, so the oracle is the library's own
    from tsplit_b200.ops.pool import np_max_pool_grad
    want = np_max_pool_grad(x.cpu().numpy(), ref_y.detach().cpu().numpy(), dy.cpu().numpy(), k, k, pad, stride)
    assert torch.equal(dx.t.cpu(), torch.from_numpy(want))


# column sums in one launch: a single row, remainders of the 32 lanes and of the four loads, ragged columns, the last row
# count; the next one takes two stages
@pytest.mark.parametrize("rows,cols", [(1, 4), (2, 33), (31, 7), (33, 64), (129, 100), (512, 1024), (513, 32)])
def test_column_sums_of_few_rows(rows, cols):
    x = _rand(rows, cols + 3)[:, :cols]
    y = torch.zeros(cols, device="cuda")
    ctx = ndarray.gpu(0)
    G.reduce_sum(x.data_ptr(), [rows, cols], [cols + 3, 1], [0], ndarray.from_tensor(y, ctx), _stream())
    # fp32 sums of at most 513 terms, sixteen or fewer of them in a row: some 30 roundings of partial sums
    bound = 32 * 2.0 ** -24 * x.double().abs().sum(0) + 1e-6
    assert torch.all((y.double() - x.double().sum(0)).abs() <= bound)
    if 1 < rows <= 512:
        items = [(ndarray.from_tensor(x.contiguous(), ctx), ndarray.from_tensor(torch.zeros(cols, device="cuda"), ctx)),
                 (ndarray.from_tensor(_rand(3, 5), ctx), ndarray.from_tensor(torch.zeros(5, device="cuda"), ctx))]
        assert G.colsum_group(items, _stream())
        assert torch.equal(items[0][1].t, y)
        torch.testing.assert_close(items[1][1].t, items[1][0].t.sum(0), rtol=0, atol=1e-6)


# rows of one vector, a lane's remainder, each register count's last and first, the longest kept row and longer ones, a
# ragged one and one that is not aligned
@pytest.mark.parametrize("d,shift", [(4, 0), (128, 0), (132, 0), (260, 0), (516, 0), (1024, 0), (1028, 0), (30, 0), (64, 1)])
@pytest.mark.parametrize("rows", [1, 77])
def test_layer_norm_gradient_of_rows(d, shift, rows):
    ctx = ndarray.gpu(0)
    flat = lambda seed: _rand(rows * d + shift, seed=seed)[shift:].view(rows, d)
    x, dy, dx = flat(1), flat(2), flat(3)
    scale = _rand(d, seed=4) + 1
    mean, inv = x.mean(1), 1 / torch.sqrt(x.var(1, unbiased=False) + 1e-5)
    ds, db = torch.zeros(d, device="cuda"), torch.zeros(d, device="cuda")
    a = lambda t: ndarray.from_tensor(t, ctx)
    G.layer_norm_grad(a(dy), a(x), a(scale), a(mean), a(inv), a(dx), a(ds), a(db), _stream())
    xd, g = x.double(), dy.double() * scale.double()
    xn = (xd - mean.double()[:, None]) * inv.double()[:, None]
    want = inv.double()[:, None] * (g - g.mean(1, keepdim=True) - xn * (g * xn).mean(1, keepdim=True))
    # a dozen fp32 roundings of terms that are at most the largest of the row
    bound = 16 * 2.0 ** -23 * inv.double()[:, None] * (g.abs().amax(1, keepdim=True) * (1 + xn.abs().amax(1, keepdim=True) ** 2))
    assert torch.all((dx.double() - want).abs() <= bound + 1e-6)


@pytest.mark.parametrize("n,vocab,dim", [(1, 3, 4), (700, 5, 512), (33, 40, 6), (64, 9, 132)])
def test_embedding_gradient_of_repeated_ids(n, vocab, dim):
    ctx = ndarray.gpu(0)
    ids = torch.randint(-1, vocab + 1, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).float()
    g = torch.round(_rand(n, dim) * 8) / 8                              # sums of eighths are exact in any order
    table = torch.zeros(vocab, dim, device="cuda")
    G.embedding_grad(ndarray.from_tensor(g, ctx), ndarray.from_tensor(ids, ctx), ndarray.from_tensor(table, ctx), _stream())
    inside = (ids >= 0) & (ids < vocab)
    assert torch.equal(table, torch.zeros_like(table).index_add_(0, ids[inside].long(), g[inside]))


@pytest.mark.parametrize("n,vocab,dim", [(1, 3, 4), (700, 5, 512), (33, 40, 6), (129, 9, 12)])
def test_embedding_rows(n, vocab, dim):
    ctx = ndarray.gpu(0)
    ids = torch.randint(-1, vocab + 1, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).float()
    table, y = _rand(vocab, dim), torch.full((n + 1, dim), 7.0, device="cuda")
    G.embedding(ndarray.from_tensor(table, ctx), ndarray.from_tensor(ids, ctx), ndarray.from_tensor(y[:n], ctx), _stream())
    inside = ((ids >= 0) & (ids < vocab))[:, None]                       # other ids give rows of zeros
    assert torch.equal(y[:n], torch.where(inside, table[ids.long().clamp(0, vocab - 1)], torch.zeros((), device="cuda")))
    assert torch.all(y[n] == 7)


@pytest.mark.parametrize("rows,cols", [(514, 4), (1023, 36), (8160, 512), (20000, 1000), (600, 16500)])
def test_column_sums_of_many_rows(rows, cols):
    x, y = _rand(rows, cols), torch.zeros(cols, device="cuda")
    G.reduce_sum(x.data_ptr(), [rows, cols], [cols, 1], [0], ndarray.from_tensor(y, ndarray.gpu(0)), _stream())
    # pairwise joins of partial sums of at most some eighty terms
    assert torch.all((y.double() - x.double().sum(0)).abs() <= 96 * 2.0 ** -24 * x.double().abs().sum(0))


# rows that stay in registers and rows that do not, at both sides of each line; four-element batches and their rest
@pytest.mark.parametrize("cols", [1, 3, 127, 129, 511, 1021, 1023, 1025, 2047, 2049])
def test_cross_entropy_of_short_and_odd_rows(cols):
    ctx, rows = ndarray.gpu(0), 37
    x, g = 3 * _rand(rows, cols), torch.full((1,), 0.5, device="cuda")
    lab = torch.softmax(_rand(rows, cols, seed=1), 1)
    a = lambda t: ndarray.from_tensor(t, ctx)
    loss, dx = torch.zeros(1, device="cuda"), torch.full((rows, cols), 9.0, device="cuda")
    G.softmax_ce(a(x), a(lab), a(loss), _stream())
    G.softmax_ce_grad(a(x), a(lab), a(g), a(dx), _stream())
    _stream().sync()
    lp = torch.log_softmax(x.double(), 1)
    # fp32 sums of at most some two thousand terms of one sign, and the exponential's 2^-21
    torch.testing.assert_close(loss[0].double(), -(lab.double() * lp).sum(1).mean(), rtol=2e-5, atol=1e-6)
    torch.testing.assert_close(dx.double(), (lp.exp() - lab.double()) * 0.5 / rows, rtol=1e-4, atol=1e-6 * 0.5 / rows)


@pytest.mark.parametrize("cols", [1, 600, 1000, 1024, 1025, 1200, 5000])
def test_softmax_rows_and_gradient(cols):
    ctx, rows = ndarray.gpu(0), 19
    x, dy = 3 * _rand(rows, cols), _rand(rows, cols, seed=1)
    a = lambda t: ndarray.from_tensor(t, ctx)
    y, dx = torch.full_like(x, 9.0), torch.full_like(x, 9.0)
    G.softmax(a(x), a(y), _stream())
    G.softmax_grad(a(y), a(dy), a(dx), _stream())
    _stream().sync()
    ref = torch.softmax(x.double(), 1)
    torch.testing.assert_close(y.double(), ref, rtol=1e-4, atol=1e-9)                  # the fast exponential's 2^-21, sums
    yd = y.double()
    torch.testing.assert_close(dx.double(), yd * (dy.double() - (yd * dy.double()).sum(1, keepdim=True)), rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("d", [1, 31, 128, 129, 512, 513, 1000, 1024, 1025, 1500])
def test_layer_norm_rows(d):
    ctx, rows = ndarray.gpu(0), 13
    x, scale, bias = _rand(rows, d) + 0.5, _rand(d, seed=1) + 1, _rand(d, seed=2)
    y, mean, inv = torch.full_like(x, 9.0), torch.zeros(rows, device="cuda"), torch.zeros(rows, device="cuda")
    a = lambda t: ndarray.from_tensor(t, ctx)
    G.layer_norm(a(x), a(scale), a(bias), a(y), a(mean), a(inv), 1e-3, _stream())
    _stream().sync()
    want = torch.nn.functional.layer_norm(x.double(), (d,), scale.double(), bias.double(), 1e-3)
    # the variance as a difference of sums of squares: some 2^-20 of the mean square, seen through 1 / sqrt(var + 1e-3)
    torch.testing.assert_close(y.double(), want, rtol=1e-4, atol=1e-3 if d == 1 else 1e-4)


@pytest.mark.parametrize("n", [1, 255, 257, 148 * 8 * 256 * 8 - 1, 148 * 8 * 256 * 9 + 3])
def test_where_and_dropout_cover_the_tensor_once(n):
    ctx = ndarray.gpu(0)
    c, p, q = (_rand(n, seed=k) for k in range(3))
    c[c < 0] = 0
    out, drop = torch.full((n + 8,), 7.0, device="cuda"), torch.full((n + 8,), 7.0, device="cuda")
    a = lambda t: ndarray.from_tensor(t, ctx)
    G.where(a(c), a(p), a(q), a(out[:n]), _stream())
    G.dropout(a(p), a(drop[:n]), 0.75, 11, _stream())
    _stream().sync()
    assert torch.equal(out[:n], torch.where(c != 0, p, q)) and torch.all(out[n:] == 7) and torch.all(drop[n:] == 7)
    from tsplit_b200.ops.misc import philox_like_mask
    keep = torch.from_numpy(philox_like_mask((n,), 0.75, 11)).cuda()
    torch.testing.assert_close(drop[:n], torch.where(keep, p / 0.75, torch.zeros_like(p)), rtol=1e-6, atol=0)


@pytest.mark.parametrize("tk", [4, 37, 128, 132, 256, 512, 516, 1000, 1024])
@pytest.mark.parametrize("keys", [True, False])
@pytest.mark.parametrize("causal", [0, 1])
def test_masked_softmax_rows(tk, keys, causal):
    n, h, tq = 2, 3, 5
    x = _rand(n, h, tq, tk)
    k = (torch.arange(tk, device="cuda")[None, :] < torch.tensor([[tk], [max(1, tk // 2)]], device="cuda")).float()
    a = lambda t: ndarray.from_tensor(t, ndarray.gpu(0))
    y = torch.full_like(x, 9.0)
    G.masked_softmax(a(x), a(k) if keys else None, a(y), 0.25, causal, _stream())
    _stream().sync()
    t = x.double() * 0.25
    if keys:
        t = t + torch.where(k == 0, -1e9, 0.0).double()[:, None, None, :]
    if causal:
        t = torch.where(torch.ones(tq, tk, device="cuda").tril() > 0, t, torch.full((), -1e9, dtype=t.dtype, device="cuda"))
    torch.testing.assert_close(y.double(), torch.softmax(t, -1), rtol=1e-4, atol=1e-8)      # the fast exponential's 2^-21


# few rows of wide arrays: the widths of the single launch and the first past them, for many rows and for few; then many
# chunks (more than 128) of few columns and of many
@pytest.mark.parametrize("rows,cols", [(64, 8192), (129, 8192), (129, 8196), (128, 16384), (128, 16388), (63, 16388), (512, 16386),
                                       (300, 65536), (2, 65536), (4127, 64), (4160, 64), (4200, 4096), (4200, 4100)])
def test_column_sums_of_wide_arrays(rows, cols):
    x, y = _rand(rows, cols), torch.zeros(cols, device="cuda")
    G.reduce_sum(x.data_ptr(), [rows, cols], [cols, 1], [0], ndarray.from_tensor(y, ndarray.gpu(0)), _stream())
    _stream().sync()
    # at most some hundred roundings of partial sums in a row
    assert torch.all((y.double() - x.double().sum(0)).abs() <= 160 * 2.0 ** -24 * x.double().abs().sum(0))


LOWEST = float(np.finfo(np.float32).min)


def _first_maximum_gradient(x, dy, k, pad, stride):
    """The first pixel of a window that nothing after it exceeds takes its gradient; comparisons with NaN are false."""
    n, c, h, w = x.shape
    dx = np.zeros_like(x)
    for b, ch, oy, ox in np.ndindex(dy.shape):
        best = None
        for iy in range(max(0, oy * stride - pad), min(h, oy * stride - pad + k)):
            for ix in range(max(0, ox * stride - pad), min(w, ox * stride - pad + k)):
                if best is None or x[b, ch, iy, ix] > x[(b, ch) + best]:
                    best = (iy, ix)
        dx[(b, ch) + best] += dy[b, ch, oy, ox]
    return dx


# one pass over tiles (with and without the constants of 3 x 3 stride 2), and two passes
@pytest.mark.parametrize("k,pad,stride", [(3, 1, 2), (2, 0, 1), (15, 7, 1)])
def test_max_pool_gradient_of_special_values(k, pad, stride):
    x = _rand(1, 4, 19, 18).cpu().numpy()
    r = np.random.RandomState(0)
    for v in (LOWEST, -np.inf, np.inf, np.nan):
        x[0, r.randint(0, 4, 30), r.randint(0, 19, 30), r.randint(0, 18, 30)] = v
    x[0, 1, :9, :9], x[0, 2, :9, :9] = LOWEST, -np.inf                       # whole windows of them
    oh, ow = (19 + 2 * pad - k) // stride + 1, (18 + 2 * pad - k) // stride + 1
    dy = np.round(_rand(1, 4, oh, ow, seed=1).cpu().numpy() * 8) / 8          # sums of eighths are exact
    t = lambda a: _arr(torch.from_numpy(a).cuda())
    dx, y = _arr(torch.full((1, 4, 19, 18), 7.0, device="cuda")), t(np.zeros((1, 4, oh, ow), np.float32))
    G.pool_grad(0, t(x), y, t(dy), dx, k, k, pad, stride, _stream())
    _stream().sync()
    np.testing.assert_array_equal(dx.t.cpu().numpy(), _first_maximum_gradient(x, dy, k, pad, stride))


@pytest.mark.parametrize("rows", [2, 63, 64, 512, 513])
def test_column_sums_of_special_values(rows):
    x = _rand(rows, 40)
    x[0, 3], x[rows - 1, 4], x[0, 5], x[rows - 1, 5] = float("inf"), float("-inf"), float("inf"), float("-inf")
    x[rows // 2, 6] = float("nan")
    x[0, 7], x[rows - 1, 7] = LOWEST, LOWEST                                  # below the range of fp32
    x[:, 8] = 0
    x[0, 8], x[rows - 1, 8] = LOWEST, -LOWEST
    y = torch.zeros(40, device="cuda")
    G.reduce_sum(x.data_ptr(), [rows, 40], [40, 1], [0], ndarray.from_tensor(y, ndarray.gpu(0)), _stream())
    _stream().sync()
    assert y[3] == float("inf") and y[4] == float("-inf") and torch.isnan(y[5]) and torch.isnan(y[6])
    assert y[7] == float("-inf") and y[8] == 0
    assert torch.isfinite(y[[0, 1, 2]]).all() and torch.isfinite(y[9:]).all()


# a block per window, several, and a thread per output
@pytest.mark.parametrize("hw", [8, 57, 7])
def test_average_pool_of_special_values(hw):
    x = _rand(2, 8, hw, hw)
    x[0, 0, 0, 0], x[0, 1, -1, -1], x[1, 2, 3, 3] = float("inf"), float("-inf"), float("nan")
    x[1, 3, 0, 0], x[1, 3, -1, -1], x[1, 4] = float("inf"), float("-inf"), 0
    x[1, 4, 0, 0] = LOWEST
    ref = x.double().mean((2, 3), keepdim=True).float()
    y = _arr(torch.zeros_like(ref))
    G.pool(1, _arr(x), y, hw, hw, 0, hw, _stream())
    _stream().sync()
    # (sums of at most some hundred terms a lane, pairwise joins)
    torch.testing.assert_close(y.t, ref, rtol=1e-5, atol=1e-5, equal_nan=True)


@pytest.mark.parametrize("d", [64, 1024, 1028, 30])
def test_layer_norm_gradient_keeps_special_values_in_their_row(d):
    ctx = ndarray.gpu(0)
    rows = 9
    x, dy, scale = _rand(rows, d, seed=1), _rand(rows, d, seed=2), _rand(d, seed=4) + 1
    mean, inv = x.mean(1), 1 / torch.sqrt(x.var(1, unbiased=False) + 1e-5)
    a = lambda t: ndarray.from_tensor(t, ctx)
    outs = []
    for v in (None, float("nan"), float("inf")):
        g = dy.clone()
        if v is not None:
            g[4, d - 1] = v
        dx, ds, db = torch.zeros_like(x), torch.zeros(d, device="cuda"), torch.zeros(d, device="cuda")
        G.layer_norm_grad(a(g), a(x), a(scale), a(mean), a(inv), a(dx), a(ds), a(db), _stream())
        _stream().sync()
        outs.append(dx)
    others = [r for r in range(rows) if r != 4]
    for dx in outs[1:]:
        assert torch.equal(dx[others], outs[0][others]) and not torch.isfinite(dx[4]).any()
