"""The native host path (csrc/host.cpp) against the Python layer on the same kernels: results and gradients
bit for bit, over operand forms, sizes at the edges of a vector and of a block, and layouts."""
import contextlib

import pytest
import torch

import pam_b200 as pam
from conftest import assert_bits_equal
from pam_b200 import _lib, fused, optim

pytestmark = pytest.mark.gpu
DEV = "cuda"


@contextlib.contextmanager
def route(python):
    """The native host path, or the Python layer as if the native one declined every call."""
    with pytest.MonkeyPatch.context() as m:
        if python:
            m.setattr(_lib, "host", lambda: None)
        yield


def both(fn, *inputs, gy_seed=5):
    """fn on copies of `inputs` through each route: outputs and the gradients of the tensor inputs."""
    results = []
    for python in (False, True):
        with route(python):
            ins = [t.detach().clone(memory_format=torch.preserve_format).requires_grad_() if isinstance(t, torch.Tensor) else t for t in inputs]
            y = fn(*ins)
            gy = torch.randn(y.shape, generator=torch.Generator(DEV).manual_seed(gy_seed), device=DEV)
            results.append([y.detach(), *torch.autograd.grad(y, [t for t in ins if isinstance(t, torch.Tensor)], gy)])
    for k, (got, want) in enumerate(zip(*results)):
        assert_bits_equal(got, want, f"output {k}")


def randn(*shape, seed=1, specials=True):
    t = torch.randn(*shape, generator=torch.Generator(DEV).manual_seed(seed), device=DEV)
    if specials and t.numel() > 8:
        flat = t.view(-1)
        flat[::7], flat[3::11], flat[5::13] = 0.0, 1e-30, 1e30
    return t


@pytest.mark.parametrize("op", [pam.mul, pam.div])
@pytest.mark.parametrize("approx", [True, False, (True, False), (False, True)])
@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1024, 1025, 2047, 2048, 2052, 6145])
def test_elementwise_sizes(op, approx, n):
    a, b = randn(n), randn(n, seed=2)
    both(lambda x, y: op(x, y, approx_bwd=approx, offset=1.0552), a, b)
    padded = randn(n + 1)
    both(lambda x, y: op(x[1:], y, approx_bwd=approx), padded, b)                 # not 16-byte aligned


@pytest.mark.parametrize("op", [pam.mul, pam.div])
@pytest.mark.parametrize("approx", [True, False])
def test_elementwise_broadcasts(op, approx):
    full = randn(6, 5, 8)
    for other in (randn(8, seed=3), randn(5, 8, seed=3), randn(6, 1, 1, seed=3), randn(6, 5, 1, seed=3), randn(1, seed=3),
                  randn(1, 5, 1, seed=3), torch.tensor(0.7, device=DEV), 0.3):
        both(lambda x, y: op(x, y, approx_bwd=approx), full, other)
        if not (op is pam.div and isinstance(other, torch.Tensor) and other.dim() == 0):
            both(lambda x, y: op(y, x, approx_bwd=approx), full, other)
    both(lambda x, y: op(x, y, approx_bwd=approx), randn(6, 1, 8), randn(1, 5, 1, seed=4))    # neither has the full shape
    both(lambda x, y: op(x.transpose(0, 1), y, approx_bwd=approx), randn(5, 6), randn(6, 5, seed=4))


@pytest.mark.parametrize("approx", [True, False])
@pytest.mark.parametrize("rows,fin,fout", [(1, 64, 64), (32, 130, 67), (197, 192, 96)])
def test_linear_and_products(approx, rows, fin, fout):
    x, w, b = randn(rows, fin), randn(fout, fin, seed=2), randn(fout, seed=3)
    # (the weight gradient is formed as [out, in] here and as [in, out] there: plans and sums are the same either way)
    for strict in (False, True):
        pam.set_strict_k_order(strict)
        both(lambda x, w, b: pam.linear(x, w, b, approx_bwd=approx), x, w, b)
        both(lambda x, w: pam.linear(x, w, approx_bwd=approx), x, w)
        both(lambda x, w, b: pam.linear(x[None].expand(3, -1, -1), w, b, approx_bwd=approx), x, w, b)
        both(lambda x, w: pam.linear(x, w.T.contiguous().T, approx_bwd=approx), x, w)
        both(lambda x, w: pam.matmul(x, w.T, approx_bwd=approx), x, w)
        both(lambda x, w: pam.matmul(x, w, approx_bwd=(approx, not approx)), x, randn(fin, fout, seed=2))
        both(lambda x, y: pam.bmm(x, y.mT, approx_bwd=approx), randn(3, rows, fin), randn(3, fout, fin, seed=2))
        both(lambda x, y: pam.bmm(x, y, approx_bwd=approx), randn(3, rows, 9)[:, :, ::2], randn(3, 5, fout, seed=2))


@pytest.fixture(autouse=True)
def default_k_order():
    yield
    pam.set_strict_k_order(False)


@pytest.mark.parametrize("approx", [True, False])
def test_rows(approx):
    x = randn(3, 7, 65, specials=False)
    w, b = randn(65, seed=2, specials=False), randn(65, seed=3, specials=False)
    both(lambda x, w, b: pam.layer_norm(x, (65,), w, b, approx_bwd=approx), x, w, b)
    both(lambda x, b: pam.layer_norm(x, (65,), None, b, approx_bwd=approx), x, b)
    both(lambda x: pam.layer_norm(x.transpose(0, 1), (65,), approx_bwd=approx), x)
    both(lambda x: pam.softmax(x, dim=-1, approx_bwd=approx), x)
    both(lambda x: pam.softmax(x.transpose(0, 1), dim=2, approx_bwd=approx), x)


@pytest.mark.parametrize("T,S,heads,hd", [(1, 1, 1, 1), (5, 7, 2, 3), (33, 17, 3, 8), (64, 130, 1, 64)])
@pytest.mark.parametrize("offset", [None, 1.0552])
def test_attention(T, S, heads, hd, offset):
    d = heads * hd
    for qkv in (randn(2, T, 3 * d, specials=False), randn(T, 2, 3 * d, specials=False).transpose(0, 1)):
        both(lambda t: fused.attention_qkv(t, heads, hd ** -0.5, offset=offset), qkv)
        with route(False):
            y = fused.attention_qkv(qkv, heads, hd ** -0.5, offset=offset)        # (no gradient: nothing is kept)
        with route(True):
            assert_bits_equal(y, fused.attention_qkv(qkv, heads, hd ** -0.5, offset=offset))
    causal = torch.full((T, S), float("-inf"), device=DEV).triu(1 + max(S - T, 0))
    for mask in (None, causal, randn(2 * heads, T, S, seed=6, specials=False)):
        both(lambda q, k, v: fused.attention_heads(q, k, v, heads, mask, offset=offset), randn(2, T, d, specials=False),
             randn(2, S, d, seed=2, specials=False), randn(S, 2, d, seed=3, specials=False).transpose(0, 1))


def test_adam_groups_and_fallbacks():
    """Two groups, a parameter without a gradient, unequal step counts; then a group that the native collection
    declines (a half-precision parameter), which steps through the dictionary of operators."""
    def run(python, half):
        with route(python):
            g = torch.Generator(DEV).manual_seed(3)
            ps = [torch.nn.Parameter(torch.randn(n, generator=g, device=DEV)) for n in (1, 5, 1024, 4099)]
            if half:
                ps.append(torch.nn.Parameter(torch.randn(17, generator=g, device=DEV).half()))
            opt = optim.Adam([{"params": ps[:2], "weight_decay": 0.1}, {"params": ps[2:]}], lr=1e-2, opt_functional_cfg="pam")
            for step in range(3):
                for k, p in enumerate(ps):
                    p.grad = None if (k == 1 and step != 1) else torch.randn(p.shape, generator=g, device=DEV).to(p.dtype)
                opt.step()
            steps = [opt.state[p]["step"] for p in ps]
            return [t for p in ps for t in (p.detach().float(), opt.state[p]["exp_avg"], opt.state[p]["exp_avg_sq"])], steps

    for half in (False, True):
        (got, steps), (want, want_steps) = run(False, half), run(True, half)
        assert steps == want_steps == [3, 1, 3, 3] + [3] * half
        for k, (u, v) in enumerate(zip(got, want)):
            assert_bits_equal(u, v, f"tensor {k}")


def test_errors_are_those_of_the_python_layer():
    x = torch.ones(2, 3, device=DEV)
    with pytest.raises(ValueError, match="inner dimensions differ"):
        pam.matmul(x, x)
    with pytest.raises(RuntimeError):
        pam.mul(x, torch.ones(4, device=DEV))
    with pytest.raises(RuntimeError):
        pam.mul(x, torch.ones(3))
    y = pam.mul(x.requires_grad_(), x)
    y.sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        y.sum().backward()


def test_nvtx_ranges_are_around_the_path_that_runs_without_them():
    x, w = randn(70, 50, specials=False).requires_grad_(), randn(30, 50, seed=2, specials=False).requires_grad_()
    plain = pam.linear(x, w, approx_bwd=True)
    pam.set_nvtx(True)
    try:
        traced = pam.linear(x, w, approx_bwd=True)
        grads = torch.autograd.grad(traced.sum(), [x, w])
    finally:
        pam.set_nvtx(False)
    assert traced.grad_fn.name() == plain.grad_fn.name() == "PamLinearBackward"
    for got, want in zip((traced, *grads), (plain, *torch.autograd.grad(plain.sum(), [x, w]))):
        assert_bits_equal(got.detach(), want.detach())
