"""Rows of a softmax whose values all lie far inside the range rules' bounds skip the rules: forward, saved exponentials and the backward pass
from them, against the same chain of elementwise kernels with the row sums in the kernel's own order, bit for bit.  Rows that
qualify, rows that do not (zeros, tiny and great values, inf, NaN, masks) and mixtures of them, at the lengths where the
layouts change, with offsets and post scales inside and outside of what the shorter form allows."""
import math

import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu

LOG2E, LN2 = float(torch.tensor(math.log2(math.e))), float(torch.tensor(math.log(2.0)))


def _row_sum(v):
    """Sums of the rows as a warp forms them: each lane its columns in order from +0, then a butterfly over the lanes."""
    rows, n = v.shape
    width = 4 if n % 4 == 0 else 1
    chunks = -(-n // (32 * width))
    padded = torch.zeros(rows, chunks * 32 * width, device=v.device)
    used = torch.zeros(chunks * 32 * width, dtype=torch.bool, device=v.device)
    padded[:, :n], used[:n] = v, True
    padded, used = padded.view(rows, chunks, 32, width), used.view(chunks, 32, width)
    s = torch.zeros(rows, 32, device=v.device)
    for q in range(chunks):
        for c in range(width):
            s = torch.where(used[q, :, c], s + padded[:, q, :, c], s)
    lane = torch.arange(32, device=v.device)
    for d in (16, 8, 4, 2, 1):
        s = s + s[:, lane ^ d]
    return s[:, :1]


def _ops(offset):
    from pam_b200.cuda_bindings import cuda_kernels as k
    full = lambda a, b: b.expand_as(a).contiguous() if isinstance(b, torch.Tensor) else torch.full_like(a, b)
    return (lambda a, b: k.pam_fwd(a, full(a, b), offset)), (lambda a, b: k.pad_fwd(a, full(a, b), offset)), (lambda a: k.pa_exp_fwd(a, 2.0, offset))


def _forward(x, offset):
    mul, div, exp2 = _ops(offset)
    masked = x == float("-inf")
    scaled = torch.where(masked, x, mul(x, LOG2E))
    e = torch.where(masked, torch.zeros_like(x), exp2(scaled - torch.floor(scaled.max())))
    return div(e, _row_sum(e)), torch.where(masked, torch.full_like(e, -0.0), e)


def _backward(e, g, offset, post):
    mul, div, _ = _ops(offset)
    masked = e.view(torch.int32) == -2 ** 31
    total = _row_sum(e)
    d = mul(g, div(torch.ones_like(total), total)) + _row_sum(-mul(div(div(e, total), total), g))
    d = torch.where(masked, torch.zeros_like(d), mul(mul(e, LN2), torch.where(masked, torch.zeros_like(d), d)))
    d = mul(d, LOG2E)
    return d if post is None else mul(d, post)


def _inputs(kind, rows, n, g):
    x, dy = torch.randn(rows, n, generator=g) * 2, torch.randn(rows, n, generator=g) * 1e-3
    some = torch.rand(rows, 1, generator=g) < 0.3
    if kind == "masked": x = x.masked_fill(torch.arange(n)[None] > (torch.arange(rows) % n)[:, None], float("-inf"))
    if kind == "zeros": x[:, n // 2], dy[:, n // 3] = 0.0, 0.0
    if kind == "mixed":
        x, dy = torch.where(some & (torch.rand(rows, n, generator=g) < 0.1), torch.zeros(()), x), torch.where(some, dy * 1e-12, dy)
        dy[some.flip(0).expand(rows, n) & (torch.rand(rows, n, generator=g) < 0.05)] = 1e25
    if kind == "wide": x, dy = x * 25, dy * torch.exp2(torch.randint(-70, 60, (rows, n), generator=g).float())
    if kind == "odd":
        x[torch.rand(rows, n, generator=g) < 0.02] = float("-inf")
        x[0] = float("-inf")
        dy[torch.rand(rows, n, generator=g) < 0.01] = float("nan")
        dy[torch.rand(rows, n, generator=g) < 0.01] = float("inf")
    if kind == "equal": x[:], dy[:] = 1.0, 0.25
    if kind == "some zeros":                                 # of either sign, among inputs and gradients, and rows of gradients that are all zeros
        x, dy = (torch.where(torch.rand(rows, n, generator=g) < 0.1, torch.tensor([0.0, -0.0])[torch.randint(0, 2, (rows, n), generator=g)], t) for t in (x, dy))
        x[1::4], dy[::5] = x[1::4] + 3.0, 0.0                # (shifts of zero and of more)
    if kind == "deep": x[:, n // 2] -= torch.arange(rows) * 2.0          # exponentials from one down to beyond the least normal number
    return x.cuda(), dy.cuda()


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 128, 197, 224, 225, 252, 255, 256, 500, 512, 700, 768, 1001, 1024])
@pytest.mark.parametrize("kind", ["plain", "masked", "zeros", "mixed", "wide", "odd", "equal", "some zeros", "deep"])
@pytest.mark.parametrize("offset,post", [(1.0, None), (1.0552, 0.125), (0.97, 1e-3), (1.5, -2.0)])
def test_rows_in_both_forms(n, kind, offset, post):
    from pam_b200 import _lib
    lib, stream = _lib.lib(), torch.cuda.current_stream().cuda_stream
    rows = 61
    x, dy = _inputs(kind, rows, n, torch.Generator().manual_seed(n))
    y, e, only, dx = (torch.full((rows, n), -7.0, device="cuda") for _ in range(4))
    ws = torch.empty(4096, device="cuda")
    _lib.check(lib.pamk_softmax_fwd_save(x.data_ptr(), y.data_ptr(), e.data_ptr(), rows, n, offset, ws.data_ptr(), 4 * ws.numel(), stream), "save")
    _lib.check(lib.pamk_softmax_fwd(x.data_ptr(), only.data_ptr(), rows, n, offset, ws.data_ptr(), 4 * ws.numel(), stream), "fwd")
    want, want_e = _forward(x, offset)
    assert_bits_equal(e, want_e, "exponentials")
    assert_bits_equal(y, want, "probabilities")
    assert_bits_equal(only, want, "probabilities alone")
    _lib.check(lib.pamk_softmax_bwd_saved(e.data_ptr(), dy.data_ptr(), dx.data_ptr(), rows, n, offset, post is not None, post or 0.0, stream), "bwd")
    assert_bits_equal(dx, _backward(e, dy, offset, post), "gradient")


def test_many_rows_per_warp():
    """More rows than warps, so that every warp meets rows of both forms in turn."""
    test_rows = 30000
    from pam_b200 import _lib
    lib, stream = _lib.lib(), torch.cuda.current_stream().cuda_stream
    x, dy = _inputs("mixed", test_rows, 40, torch.Generator().manual_seed(3))
    y, e, dx = (torch.empty_like(x) for _ in range(3))
    ws = torch.empty(4096, device="cuda")
    _lib.check(lib.pamk_softmax_fwd_save(x.data_ptr(), y.data_ptr(), e.data_ptr(), test_rows, 40, 1.0, ws.data_ptr(), 4 * ws.numel(), stream), "save")
    _lib.check(lib.pamk_softmax_bwd_saved(e.data_ptr(), dy.data_ptr(), dx.data_ptr(), test_rows, 40, 1.0, 0, 0.0, stream), "bwd")
    want, want_e = _forward(x, 1.0)
    assert_bits_equal(e, want_e), assert_bits_equal(y, want)
    assert_bits_equal(dx, _backward(e, dy, 1.0, None))


@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("offset", [1.0, 1.0552])
def test_great_exponentials_whose_gradient_cancels(n, offset):
    """Exponentials of a caller's own, far above those that the forward pass saves, with gradients that cancel: e * 0 is +0."""
    from pam_b200 import _lib
    k = torch.arange(-60, 61, dtype=torch.float32)
    e, dy = torch.exp2(k)[:, None].expand(-1, n).contiguous().cuda(), torch.ones(121, n, device="cuda")
    e, dy = torch.cat([e, e * 1.5, e]), torch.cat([dy, dy, dy * 2.0 ** -20])
    dx = torch.full_like(e, -7.0)
    _lib.check(_lib.lib().pamk_softmax_bwd_saved(e.data_ptr(), dy.data_ptr(), dx.data_ptr(), e.shape[0], n, offset, 0, 0.0,
                                                 torch.cuda.current_stream().cuda_stream), "bwd")
    assert_bits_equal(dx, _backward(e, dy, offset, None))
