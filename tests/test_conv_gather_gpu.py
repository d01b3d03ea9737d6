"""The gathering convolution kernels at the edges of their bookkeeping, against 64-bit torch on operands cut to TF32."""
import ctypes

import pytest
import torch

from tsplit_b200 import _base

pytestmark = pytest.mark.gpu

PTR = ctypes.c_void_p


def _rand(*shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(shape, generator=g, device="cuda")
    return (x.view(torch.int32) & -8192).view(torch.float32)        # what the tensor cores read of it


# channels of no 32; a k-block of eight taps, of parts of two, of one tap; 64 filter taps (one mask) and 81 (none); filters
# wider than the image, padding of more than the image's width, images of fewer pixels than a thread's step, strides
@pytest.mark.parametrize("n,c,h,w,o,kh,kw,ph,pw,stride", [
    (2, 4, 40, 36, 64, 7, 7, 3, 3, 2), (2, 20, 9, 11, 12, 5, 5, 2, 2, 1), (1, 36, 13, 6, 20, 8, 8, 7, 7, 1),
    (2, 8, 12, 11, 12, 9, 9, 4, 4, 1), (3, 100, 5, 3, 68, 3, 3, 1, 1, 1), (7, 12, 2, 2, 36, 1, 3, 0, 1, 1),
    (2, 44, 15, 17, 60, 3, 1, 1, 0, 2), (300, 4, 1, 1, 8, 1, 1, 0, 0, 1), (1, 24, 33, 130, 12, 1, 7, 0, 6, 3)])
def test_forward_and_gradients(n, c, h, w, o, kh, kw, ph, pw, stride):
    _check(n, c, h, w, o, kh, kw, ph, pw, stride)


# both channel counts multiples of 32, where the data gradient reads the filters in place: one tile, ragged tiles, CTA pairs,
# filters larger than the padding, a pointwise and an asymmetric one, the four parities of stride 2
# (which write their pixels of dx: tiles that cross rows and images, several to a CTA, classes without rows or taps)
@pytest.mark.parametrize("n,c,h,w,o,kh,kw,ph,pw,stride", [
    (2, 32, 9, 9, 32, 3, 3, 1, 1, 1), (3, 96, 17, 19, 64, 5, 3, 2, 0, 1), (4, 320, 60, 61, 64, 3, 3, 1, 1, 1),
    (4, 256, 50, 47, 96, 1, 1, 0, 0, 1), (2, 224, 17, 17, 192, 1, 7, 0, 3, 1), (2, 32, 9, 9, 32, 7, 7, 3, 3, 2),
    (3, 96, 17, 20, 64, 5, 5, 2, 2, 2), (8, 512, 28, 28, 128, 1, 1, 0, 0, 2),
    (24, 256, 56, 55, 32, 3, 3, 1, 1, 2), (5, 288, 33, 31, 32, 2, 3, 0, 1, 2), (2, 32, 1, 9, 32, 1, 1, 0, 0, 2)])
def test_data_gradient_from_filters_in_place(n, c, h, w, o, kh, kw, ph, pw, stride):
    _check(n, c, h, w, o, kh, kw, ph, pw, stride)


def _check(n, c, h, w, o, kh, kw, ph, pw, stride):
    oh, ow = (h + 2 * ph - kh) // stride + 1, (w + 2 * pw - kw) // stride + 1
    x, wt, dy = _rand(n, h, w, c, seed=1), _rand(o, kh, kw, c, seed=2), _rand(n, oh, ow, o, seed=3)
    xd, wd, dyd = x.double().permute(0, 3, 1, 2), wt.double().permute(0, 3, 1, 2), dy.double().permute(0, 3, 1, 2)
    lib, st = _base.kernels(), PTR(torch.cuda.current_stream().cuda_stream)
    refs = [torch.nn.functional.conv2d(xd, wd, stride=stride, padding=(ph, pw)),
            torch.nn.grad.conv2d_input(xd.shape, wd, dyd, stride=stride, padding=(ph, pw)),
            torch.nn.grad.conv2d_weight(xd, wd.shape, dyd, stride=stride, padding=(ph, pw))]
    for kind, (shape, terms) in enumerate((((n, oh, ow, o), kh * kw * c), ((n, h, w, c), kh * kw * o), ((o, kh, kw, c), n * oh * ow))):
        args = [x, wt, dy]
        args[(2, 0, 1)[kind]] = out = torch.full(shape, 7.0, device="cuda")
        rc = lib.tsb_conv2d(kind, *[PTR(a.data_ptr()) for a in args], n, c, h, w, o, kh, kw, oh, ow, ph, pw, stride, st)
        assert rc == 0, _base.error_string(rc)
        # products of 10-bit operands are exact in fp32; sums round (or truncate) once per term: 2^-23 of sums whose
        # magnitude grows as the root of their number, and no more than that root below the largest
        err = (out.double().permute(0, 3, 1, 2) - refs[kind]).abs().max().item()
        assert err <= 2 ** -23 * terms * max(refs[kind].abs().max().item(), 1.0), (kind, err)
    assert lib.tsb_device_status(st) == 0


# classes without taps, all four with some, ragged tiles and several per CTA; channels of no 32, which it leaves alone
@pytest.mark.parametrize("n,c,h,w,o,kh,kw,ph,pw", [(2, 32, 9, 9, 32, 1, 1, 0, 0), (3, 96, 17, 20, 64, 3, 3, 1, 1),
                                                   (24, 256, 56, 55, 32, 1, 1, 0, 0), (2, 100, 9, 9, 32, 1, 1, 0, 0)])
def test_strided_data_gradient_added_to_another(n, c, h, w, o, kh, kw, ph, pw):
    oh, ow = (h + 2 * ph - kh) // 2 + 1, (w + 2 * pw - kw) // 2 + 1
    wt, dy, first = _rand(o, kh, kw, c, seed=2), _rand(n, oh, ow, o, seed=3), _rand(n, h, w, c, seed=4)
    lib, st = _base.kernels(), PTR(torch.cuda.current_stream().cuda_stream)
    alone, both = torch.empty_like(first), first.clone()
    assert lib.tsb_conv2d(1, *[PTR(a.data_ptr()) for a in (alone, wt, dy)], n, c, h, w, o, kh, kw, oh, ow, ph, pw, 2, st) == 0
    rc = lib.tsb_conv2d_dgrad_add(*[PTR(a.data_ptr()) for a in (both, wt, dy)], n, c, h, w, o, kh, kw, oh, ow, ph, pw, st)
    assert rc == (2 if c % 32 else 0)
    assert torch.equal(both, first if c % 32 else first + alone)           # one addition, rounded once either way
