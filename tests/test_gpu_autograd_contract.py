"""What torch.autograd.Function promises and the native host path has to keep: tracing records the operator, forward-mode
AD and functorch transforms are refused, exceptions keep their type, missing gradients count as zeros, a compiled
backward pass runs.  Each test failed on a host path that went past one of these."""
import threading
import time

import numpy as np
import pytest
import torch
import torch.autograd.forward_ad as fwAD
from torch.utils.checkpoint import checkpoint

import pam_b200 as pam
from conftest import assert_bits_equal
from pam_b200 import _lib, cuda_bindings, fused, optim

pytestmark = pytest.mark.gpu
DEV = "cuda"


def randn(*shape, seed=1):
    return torch.randn(*shape, generator=torch.Generator(DEV).manual_seed(seed), device=DEV)


# every operator of the host path as a function of one [2, 4, 12] tensor
W = GAIN = None
OPERATORS = {
    "mul": lambda t: pam.mul(t, GAIN, approx_bwd=True),
    "mul_number": lambda t: pam.mul(2.5, t, approx_bwd=True),
    "div": lambda t: pam.div(t, 3.0, approx_bwd=True),
    "linear": lambda t: pam.linear(t, W, GAIN[:6].contiguous(), approx_bwd=True),
    "matmul": lambda t: pam.matmul(t[0], W.T, approx_bwd=True),
    "bmm": lambda t: pam.bmm(t, t.mT, approx_bwd=True),
    "layer_norm": lambda t: pam.layer_norm(t, (12,), GAIN, GAIN, approx_bwd=True),
    "softmax": lambda t: pam.softmax(t, dim=-1, approx_bwd=True),
    "attention_qkv": lambda t: fused.attention_qkv(t, 2, 0.5),
    "attention_heads": lambda t: fused.attention_heads(t, t, t, 2),
}
each_operator = pytest.mark.parametrize("name", OPERATORS)


@pytest.fixture(autouse=True, scope="module")
def constants():
    global W, GAIN
    W, GAIN = randn(6, 12, seed=2), randn(12, seed=3)


@pytest.mark.parametrize("name", [n for n in OPERATORS if n != "attention_qkv"])     # (its function refuses traced sizes)
def test_a_trace_holds_the_operator_and_not_its_result(name):
    op = OPERATORS[name]
    with torch.no_grad():
        traced = torch.jit.trace(lambda t: op(t) + 1, randn(2, 4, 12), check_trace=False)
        x = randn(2, 4, 12, seed=9)
        assert_bits_equal(traced(x), op(x) + 1, name)


@each_operator
def test_forward_mode_is_refused(name):
    with fwAD.dual_level():
        dual = fwAD.make_dual(randn(2, 4, 12), randn(2, 4, 12, seed=4))
        with pytest.raises(NotImplementedError, match="jvp"):
            OPERATORS[name](dual)
    with torch.no_grad(), fwAD.dual_level():
        dual = fwAD.make_dual(randn(2, 4, 12), randn(2, 4, 12, seed=4))
        with pytest.raises(NotImplementedError, match="jvp"):
            OPERATORS[name](dual)


@each_operator
def test_functorch_transforms_are_refused(name):
    x, op = randn(2, 4, 12), OPERATORS[name]
    for call in (lambda: torch.func.grad(lambda t: op(t).sum())(x), lambda: torch.func.vmap(op)(x[None]),
                 lambda: torch.func.vmap(lambda s: op(x) * s)(torch.ones(2, device=DEV))):     # (x is no wrapper here)
        with pytest.raises(RuntimeError, match="setup_context"):
            call()


def test_dispatch_modes_and_subclasses_take_the_python_layer():
    from torch.utils._python_dispatch import TorchDispatchMode

    class Count(TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            Count.seen += 1
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    x = randn(5)
    with Count():
        y = pam.mul(x, 2.0)
    assert Count.seen > 0
    assert_bits_equal(y, pam.mul(x, 2.0))
    assert_bits_equal(pam.mul(x.as_subclass(Sub), 2.0), y)


@each_operator
def test_checkpointed_block_ending_in_an_operator(name):
    op = OPERATORS[name]
    grads = []
    for run in (lambda t: op(torch.tanh(t)), lambda t: checkpoint(lambda u: op(torch.tanh(u)), t, use_reentrant=False)):
        x = randn(2, 4, 12).requires_grad_()
        y = run(x)
        grads.append(torch.autograd.grad(y, x, randn(*y.shape, seed=5))[0])
    assert_bits_equal(*grads)


class _Mine(Exception):
    pass


def _raise(message):
    raise _Mine(message)


def test_exceptions_keep_their_type():
    x = randn(3).requires_grad_()
    with pytest.raises(_Mine, match="pack"):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: _raise("pack"), lambda t: t):
            pam.mul(x, 2.0)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: _raise("unpack")):
        y = pam.mul(x, 2.0)
    with pytest.raises(_Mine, match="unpack"):
        y.sum().backward()
    with pytest.raises(torch.cuda.OutOfMemoryError):                      # (4 TiB of output: refused by the allocator)
        pam.mul(torch.ones(1, device=DEV).expand(1 << 40), 2.0)
    # a product of more row tiles than a grid holds is refused by the kernel library: here only the gradient's is one
    a, b = torch.ones(1, 65535 * 128 + 1, device=DEV), torch.ones(65535 * 128 + 1, 1, device=DEV, requires_grad=True)
    with pytest.raises(_lib.PamKernelError):
        pam.matmul(b.detach(), a[:, :1].contiguous(), approx_bwd=True)
    y = pam.matmul(a, b, approx_bwd=True)
    with pytest.raises(_lib.PamKernelError):
        y.sum().backward()


def test_unpack_hooks_run_in_the_grad_mode_of_the_backward_pass():
    x, seen = randn(3).requires_grad_(), []

    def unpack(t):
        seen.append(torch.is_grad_enabled())
        return t
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        y = pam.mul(x, 2.0, approx_bwd=True)
    torch.autograd.grad(y.sum(), x, retain_graph=True)
    torch.autograd.grad(y.sum(), x, create_graph=True)
    assert seen == [False, True]


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, t):
        return t.clone()

    @staticmethod
    def backward(ctx, g):
        return None


@each_operator
def test_a_missing_gradient_counts_as_zeros(name):
    x = randn(2, 4, 12).requires_grad_()
    (grad,) = torch.autograd.grad(_NoGradient.apply(OPERATORS[name](x)).sum(), x)
    assert grad.shape == x.shape and bool((grad == 0).all())


@each_operator
def test_compiled_autograd(name):
    from torch._dynamo import compiled_autograd
    op = OPERATORS[name]
    for seed, scale in ((1, 1.0), (2, 3.0)):
        x = randn(2, 4, 12, seed=seed).requires_grad_()
        y = op(x * scale)
        gy = randn(*y.shape, seed=5)
        (want,) = torch.autograd.grad(y, x, gy, retain_graph=True)
        with compiled_autograd._enable(lambda gm: torch.compile(gm, backend="eager")):
            y.backward(gy)
        assert_bits_equal(x.grad, want, name)


def test_compiled_autograd_tells_settings_apart():
    """The same graph with another number, offset or gradient mode must not run an earlier one's compiled backward pass."""
    from torch._dynamo import compiled_autograd
    for approx in (True, False):
        for offset in (None, 1.0552):
            for number in (2.0, 3.3):
                x = randn(2, 4, 12).requires_grad_()
                y = pam.softmax(pam.mul(pam.layer_norm(x, (12,), GAIN, GAIN, offset=offset, approx_bwd=approx), number, offset=offset, approx_bwd=approx),
                                dim=-1, offset=offset, approx_bwd=approx)
                gy = randn(*y.shape, seed=5)
                (want,) = torch.autograd.grad(y, x, gy, retain_graph=True)
                with compiled_autograd._enable(lambda gm: torch.compile(gm, backend="eager")):
                    y.backward(gy)
                assert_bits_equal(x.grad, want, f"{approx} {offset} {number}")


def test_pam_linear_binding_takes_matrices_only():
    with pytest.raises(ValueError, match="target_dim=2"):
        cuda_bindings.pam_linear(randn(2, 4, 12), W, GAIN[:6].contiguous())


# ---- Adam -------------------------------------------------------------------------------------------------------

def _adam(**kw):
    ps = [torch.nn.Parameter(randn(n, seed=n)) for n in (5, 1024, 33)]
    opt = optim.Adam(ps, opt_functional_cfg="pam", **kw)
    for p in ps:
        p.grad = randn(p.numel(), seed=p.numel() + 1)
        opt.state[p] = {"step": 3, "exp_avg": 0.1 * p.grad, "exp_avg_sq": 0.01 * p.grad.square()}
    return ps, opt


@pytest.mark.parametrize("number", [np.float32, np.float64, torch.tensor, lambda v: torch.tensor(v, device=DEV)])
def test_adam_takes_any_number(number, monkeypatch):
    """The native collection against the Python layer's, whose ctypes call converts whatever has a float value."""
    results = []
    for python in (False, True):
        with monkeypatch.context() as m:
            if python:
                m.setattr(_lib, "host", lambda: None)
            ps, opt = _adam(lr=number(1e-3), eps=number(1e-8), weight_decay=number(0.1))
            opt.step()
            results.append([t for p in ps for t in (p.detach(), opt.state[p]["exp_avg"], opt.state[p]["exp_avg_sq"])])
    for got, want in zip(*results):
        assert_bits_equal(got, want)


def test_adam_counts_a_step_when_it_was_taken():
    ps, opt = _adam(lr=1e-3, eps="1e-8")
    with pytest.raises(TypeError):
        opt.step()
    assert [opt.state[p]["step"] for p in ps] == [3, 3, 3]
    opt.param_groups[0]["eps"] = 1e-8
    opt.step()
    assert [opt.state[p]["step"] for p in ps] == [4, 4, 4]


@pytest.mark.filterwarnings("ignore:optimizer contains a parameter group with duplicate")
def test_adam_takes_a_parameter_listed_twice_in_turn():
    def run(twice):
        p = torch.nn.Parameter(randn(1 << 20))
        opt = optim.Adam([p, p] if twice else [p], lr=1e-2, opt_functional_cfg="pam")
        p.grad = randn(1 << 20, seed=2)
        opt.state[p] = {"step": 0, "exp_avg": torch.zeros_like(p), "exp_avg_sq": torch.zeros_like(p)}
        for _ in range(1 if twice else 2):
            opt.step()
        return p.detach(), opt.state[p]
    (got, s), (want, t) = run(True), run(False)
    assert s["step"] == t["step"] == 2
    assert_bits_equal(got, want)
    assert_bits_equal(s["exp_avg"], t["exp_avg"])


# ---- threads and streams ------------------------------------------------------------------------------------------

def test_threads_and_streams_agree():
    """The same block, forward and backward, from four threads on a stream each, repeatedly, against one thread's."""
    def block(x, w, g):
        y = pam.softmax(pam.layer_norm(pam.linear(x, w, g, approx_bwd=True), (64,), g, g, approx_bwd=True), dim=-1, approx_bwd=True)
        return torch.autograd.grad(pam.mul(y, y, approx_bwd=True).sum(), [x, w, g])
    data = [(randn(300, 128, seed=k).requires_grad_(), (randn(64, 128, seed=k + 10) * 0.1).requires_grad_(),
             randn(64, seed=k + 20).requires_grad_()) for k in range(4)]
    want = [block(*d) for d in data]
    torch.cuda.synchronize()
    got, errors = [None] * 4, []

    def work(k):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(20):
                    got[k] = block(*data[k])
            stream.synchronize()
        except Exception as e:                                # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            assert_bits_equal(a, b)


def test_python_threads_go_on_while_a_launch_waits():
    """Launches behind a busy stream: when the queue is full the launching thread waits, and only that thread may."""
    x = randn(8)
    pam.mul(x, 2.0)
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.wait(0.005):
            ticks.append(time.perf_counter())
    ticker = threading.Thread(target=tick)
    ticker.start()
    try:
        torch.cuda._sleep(1_500_000_000)                      # (most of a second; a full queue is some 1000 launches)
        begin = time.perf_counter()
        for _ in range(3000):
            pam.mul(x, 2.0)
        waited = time.perf_counter() - begin
        torch.cuda.synchronize()
    finally:
        stop.set()
        ticker.join()
    gaps = [b - a for a, b in zip(ticks, ticks[1:])]
    assert waited > 0.3 and max(gaps) < 0.5 * waited, (waited, max(gaps))
