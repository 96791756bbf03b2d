"""The fused Adam kernel's whole blocks (1024 elements) and their ends: tensors around multiples of a block and of the
parts that a thread takes, aligned and one float off, ordinary values beside zeros, bit for bit against the oracle's step."""
import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu

SIZES = (1, 3, 4, 1023, 1024, 1025, 2047, 2048, 2049, 3072, 3075, 4096, 4100, 6145)


@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "one float off"])
@pytest.mark.parametrize("zeros", [0.0, 0.1])
@pytest.mark.parametrize("decay", [0.0, 0.05])
def test_block_edges(shift, zeros, decay, oracle):
    import ctypes

    from pam_b200 import _lib
    g = torch.Generator().manual_seed(int(zeros * 10) + shift)
    cpu = []
    for n in SIZES:
        p, gr, m, v = torch.randn(n, generator=g) * 0.05, torch.randn(n, generator=g) * 1e-3, torch.randn(n, generator=g) * 1e-4, torch.rand(n, generator=g) * 1e-6
        gr = torch.where(torch.rand(n, generator=g) < zeros, torch.zeros(()), gr)
        cpu.append((p, gr, m, v))
    def device(t):
        buf = torch.full((t.numel() + 8,), -7.0, device="cuda")
        buf[shift:shift + t.numel()] = t.cuda()
        return buf
    dev = [tuple(device(t) for t in ts) for ts in cpu]
    b1, b2, lr, eps, step = 0.9, 0.98, 1e-3, 1e-8, 3
    step_size = lr * (1 - b2 ** step) ** 0.5 / (1 - b1 ** step)
    ptrs = [(ctypes.c_void_p * len(SIZES))(*[ts[k].data_ptr() + 4 * shift for ts in dev]) for k in range(4)]
    _lib.check(_lib.lib().pamk_adam_step(*ptrs, (ctypes.c_int64 * len(SIZES))(*SIZES), len(SIZES), b1, 1 - b1, b2, 1 - b2, eps, decay * lr, step_size,
                                         1.0, torch.cuda.current_stream().cuda_stream), "adam")
    for n, ts, (p, gr, m, v) in zip(SIZES, dev, cpu):
        new_p, new_m, new_v = oracle.adam_step(p, gr, m, v, step=step, lr=lr, betas=(b1, b2), eps=eps, weight_decay=decay)
        for k, want in ((0, new_p), (2, new_m), (3, new_v), (1, gr)):
            assert_bits_equal(ts[k][shift:shift + n], want, f"{n} elements, operand {k}")
            assert bool((ts[k][:shift] == -7.0).all()) and bool((ts[k][shift + n:] == -7.0).all())


@pytest.mark.parametrize("offset", [1.0, 1.0552])
@pytest.mark.parametrize("steady", [False, True])
def test_second_moments_around_powers_of_two(offset, steady):
    """Where log2f of the second moment may round across a power of two: two million values, a few thousand of them with a mantissa
    within 2^-11 of either end, against the same rule as a chain of elementwise kernels on the device (the host's log2f may differ)."""
    import ctypes

    from pam_b200 import _lib
    from pam_b200.cuda_bindings import cuda_kernels as k
    n = 1 << 21
    g = torch.Generator(device="cuda").manual_seed(11)
    p, gr, m = (torch.randn(n, device="cuda", generator=g) * s for s in (0.05, 1e-3, 1e-4))
    v = gr.square() if steady else torch.rand(n, device="cuda", generator=g) * 1e-6
    if steady:
        ends = torch.exp2(torch.randint(-30, -15, (n // 4,), device="cuda", generator=g).float()) * (1.0 + torch.randint(-8, 9, (n // 4,), device="cuda", generator=g) * 2.0 ** -23)
        v[: n // 4], gr[: n // 4] = ends, ends.sqrt()
    mul = lambda a, b: k.pam_fwd(a, b if isinstance(b, torch.Tensor) else torch.full_like(a, b), offset)
    b1, b2, step_size, eps = 0.9, 0.98, 4e-4, 1e-8
    m1, v1 = mul(m, b1) + mul(gr, 1 - b1), mul(v, b2) + mul(mul(gr, gr), 1 - b2)
    mant = v1.view(torch.int32) & 0x7fffff
    assert int(((mant < 0x1000) | (mant >= 0x7ff000)).sum()) > 1000
    den = k.pa_exp_fwd(mul(k.pa_log_fwd(v1, 2.0, offset), 0.5), 2.0, offset) + eps
    want = p - mul(k.pad_fwd(m1, den, offset), step_size)
    ptr = lambda t: (ctypes.c_void_p * 1)(t.data_ptr())
    _lib.check(_lib.lib().pamk_adam_step(ptr(p), ptr(gr), ptr(m), ptr(v), (ctypes.c_int64 * 1)(n), 1, b1, 1 - b1, b2, 1 - b2, eps, 0.0, step_size, offset,
                                         torch.cuda.current_stream().cuda_stream), "adam")
    assert_bits_equal(m, m1), assert_bits_equal(v, v1), assert_bits_equal(p, want)
