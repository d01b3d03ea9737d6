"""Products whose blocks are all resident at once (gemm_small.cu) against the general tcgen05 path: the same bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

I64, PTR = ctypes.c_longlong, ctypes.c_void_p


def _lib():
    from tsplit_b200 import _base
    return _base.kernels()


def _stream():
    return PTR(torch.cuda.current_stream().cuda_stream)


def _ranges(m, n, k):
    """K ranges that both paths add up (choose_splits of gemm_tcgen05.cu)."""
    bn = 256 if n > 128 else 128 if n > 64 else 64
    tiles, kb = -(-m // 128) * -(-n // bn), -(-k // 32)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 1 if tiles >= sms or kb < 16 else max(1, min(sms // tiles, kb // 8, 32))


def _matrix(rows, cols, ld, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((rows, ld), device="cuda", generator=g)


# one element; one K step and a part of one; ragged tiles; rows that TMA cannot read on either side; the last sum that
# is one range and the first that is two; the longest (eight ranges, then sixteen k-blocks in one range); a whole wave
SIZES = [(1, 1, 1), (64, 32, 8), (65, 33, 13), (64, 10, 256), (256, 10, 64), (111, 128, 37), (37, 37, 32), (130, 500, 111),
         (128, 128, 511), (128, 128, 512), (32, 1000, 2048), (100, 40, 513), (64, 64, 1000), (1024, 256, 256), (7, 260, 480)]


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", SIZES)
def test_bits_of_the_general_path(m, n, k, ta, tb):
    lib = _lib()
    for pa, pb, pc in ((0, 0, 0), (1, 4, 5)):                  # dense rows; rows with gaps, of any length
        ra, ca = (k, m) if ta else (m, k)
        rb, cb = (n, k) if tb else (k, n)
        a, b = _matrix(ra, ca, ca + pa, 1), _matrix(rb, cb, cb + pb, 2)
        c = _matrix(m, n, n + pc, 3)
        before, want = c.clone(), torch.empty((m, n), device="cuda")
        strides = (I64(ca + pa), I64(cb + pb))
        rc = lib.tsb_gemm_tf32_splitk(PTR(a.data_ptr()), PTR(b.data_ptr()), PTR(want.data_ptr()), m, n, k, *strides, I64(n),
                                      ta, tb, _ranges(m, n, k), _stream())
        assert rc == 0
        for accumulate in (0, 1):
            rc = lib.tsb_gemm_tf32(PTR(a.data_ptr()), PTR(b.data_ptr()), PTR(c.data_ptr()), m, n, k, *strides, I64(n + pc),
                                   ta, tb, 1, I64(0), I64(0), I64(0), accumulate, _stream())
            assert rc == 0
            assert torch.equal(c[:, :n], want if not accumulate else want + want)
        assert torch.equal(c[:, n:], before[:, n:])            # nothing behind the columns
    assert lib.tsb_device_status(_stream()) == 0


def test_no_store_behind_the_columns_of_the_general_path():
    lib = _lib()
    m, n, k, ldc = 300, 1023, 64, 1024                         # more tiles than are resident at once
    a, b, c = _matrix(m, k, k, 1), _matrix(n, k, k, 2), _matrix(m, n, ldc, 3)
    before = c.clone()
    a, m = a.repeat(8, 1), 8 * m
    c, before = c.repeat(8, 1), before.repeat(8, 1)
    rc = lib.tsb_gemm_tf32(PTR(a.data_ptr()), PTR(b.data_ptr()), PTR(c.data_ptr()), m, n, k, I64(k), I64(k), I64(ldc), 0, 1, 1,
                           I64(0), I64(0), I64(0), 0, _stream())
    assert rc == 0
    assert torch.equal(c[:, n:], before[:, n:])
    ref = a.double() @ b.double().t()
    assert (c[:, :n].double() - ref).norm() < 1e-3 * ref.norm()          # operands are cut to 10 bits


@pytest.mark.parametrize("heads,rows,keys,d", [(4, 37, 30, 32), (2, 64, 64, 64), (3, 7, 33, 32)])
def test_batches_and_head_layout(heads, rows, keys, d):
    """Scores and context of attention: every matrix has the bits of the same product by itself."""
    lib, n = _lib(), 3
    q, kv = _matrix(n * rows, heads * d, heads * d, 1), _matrix(n * keys, heads * d, heads * d, 2)
    s, o = torch.zeros((n, heads, rows, keys), device="cuda"), torch.zeros((n * rows, heads * d), device="cuda")
    ld = I64(heads * d)
    assert lib.tsb_gemm_tf32_heads(PTR(q.data_ptr()), PTR(kv.data_ptr()), PTR(s.data_ptr()), rows, keys, d, ld, ld, I64(keys),
                                   0, 1, n * heads, I64(d), I64(d), I64(rows * keys), 0, heads, 3, _stream()) == 0
    assert lib.tsb_gemm_tf32_heads(PTR(s.data_ptr()), PTR(kv.data_ptr()), PTR(o.data_ptr()), rows, d, keys, I64(keys), ld, ld,
                                   0, 0, n * heads, I64(rows * keys), I64(d), I64(d), 0, heads, 6, _stream()) == 0
    for b in range(n):
        for h in range(heads):
            qm = q[b * rows:(b + 1) * rows, h * d:(h + 1) * d].contiguous()
            km = kv[b * keys:(b + 1) * keys, h * d:(h + 1) * d].contiguous()
            sm, om = torch.empty((rows, keys), device="cuda"), torch.empty((rows, d), device="cuda")
            assert lib.tsb_gemm_tf32_splitk(PTR(qm.data_ptr()), PTR(km.data_ptr()), PTR(sm.data_ptr()), rows, keys, d, I64(d),
                                            I64(d), I64(keys), 0, 1, 1, _stream()) == 0
            assert torch.equal(s[b, h], sm)
            assert lib.tsb_gemm_tf32_splitk(PTR(sm.data_ptr()), PTR(km.data_ptr()), PTR(om.data_ptr()), rows, d, keys, I64(keys),
                                            I64(d), I64(d), 0, 0, 1, _stream()) == 0
            assert torch.equal(o[b * rows:(b + 1) * rows, h * d:(h + 1) * d], om)
    assert lib.tsb_device_status(_stream()) == 0


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(512, 2048, 4 * 32 * 32), (1024, 1000, 9000), (2016, 1056, 2112)])
def test_long_ranges_on_pairs_have_the_bits_of_single_tiles(monkeypatch, m, n, k, ta, tb):
    """K ranges of 32 k-blocks and more run on CTA pairs: whole tiles, ragged columns, a ragged last range."""
    lib = _lib()
    a, b = _matrix(k if ta else m, m if ta else k, m if ta else k, 1), _matrix(n if tb else k, k if tb else n, k if tb else n, 2)
    c = [_matrix(m, n, n, 3) for _ in range(2)]
    for pair, out in zip(("1", "0"), c):
        monkeypatch.setenv("TSB_GEMM_PAIR", pair)
        for accumulate in (0, 1):
            assert lib.tsb_gemm_tf32(PTR(a.data_ptr()), PTR(b.data_ptr()), PTR(out.data_ptr()), m, n, k, I64(a.shape[1]),
                                     I64(b.shape[1]), I64(n), ta, tb, 1, I64(0), I64(0), I64(0), accumulate, _stream()) == 0
    assert torch.equal(*c)
    ref = (a.double().t() if ta else a.double()) @ (b.double().t() if tb else b.double())
    assert (c[0].double() - 2 * ref).norm() < 2e-3 * ref.norm()          # operands are cut to 10 bits
    assert lib.tsb_device_status(_stream()) == 0
