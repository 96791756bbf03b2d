"""Integer adds that the products' kernels form as a maximum (x + y against INT32_MIN) or as a multiply-add (x * 1 + y): equal to the
plain add for every pair of patterns, also where the sum wraps around or is INT32_MIN itself, the pattern of -0.0.  An
offset far from one brings in-band operands there: with 2^-20 the product of 2^-53 and -2^-54 has that pattern."""
import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 2, 3, 4], ids=["tile128", "tile64", "tile32", "tile112"])
def tile(request):
    import pam_b200 as pam
    from pam_b200 import _lib
    _lib.check(_lib.lib().pamk_test_set_tile_policy(request.param), "tile policy")
    pam.set_strict_k_order(True)
    yield request.param
    pam.set_strict_k_order(False)
    _lib.lib().pamk_test_set_tile_policy(0)


def _around(exponent, g, *shape):
    """+-2^exponent, every third one a few floats further up, every fifth one of ordinary size: all in the band."""
    t = torch.full(shape, 2.0 ** exponent)
    t = torch.where(torch.rand(*shape, generator=g) < 0.5, t, -t)
    bits = t.view(torch.int32) + (torch.rand(*shape, generator=g) < 0.33).int() * torch.randint(0, 4, shape, generator=g, dtype=torch.int32)
    return torch.where(torch.rand(*shape, generator=g) < 0.2, torch.randn(*shape, generator=g) + 3.0, bits.view(torch.float32))


@pytest.mark.parametrize("offset,ea,eb", [(2.0 ** -20, -53, -54), (2.0 ** 20, 50, 59), (2.0 ** -60, -20, -47), (1.0, 0, 0)])
@pytest.mark.parametrize("M,K,N", [(65, 33, 77), (116, 36, 132)], ids=["scalar loads", "128-bit loads"])
def test_sums_that_wrap(tile, offset, ea, eb, M, K, N, oracle):
    from pam_b200.cuda_bindings import cuda_kernels
    g = torch.Generator().manual_seed(M + ea)
    A, B = _around(ea, g, M, K), _around(eb, g, K, N)
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, offset)
    for x in (A.cuda(), A.cuda().t().contiguous().t()):
        for y in (B.cuda(), B.cuda().t().contiguous().t()):
            assert_bits_equal(cuda_kernels.pam_matmul_fwd(x, y, True, True, offset), want)


@pytest.mark.parametrize("delta_l", [True, False])
@pytest.mark.parametrize("M,K,N", [(65, 33, 77), (116, 36, 132)], ids=["scalar loads", "128-bit loads"])
def test_slopes_that_wrap(tile, delta_l, M, K, N, oracle):
    """The slope's pattern is an operand's plus a mantissa: the operands cover every exponent, both zeros and the ends of the range."""
    from pam_b200 import cuda_bindings as cb
    g = torch.Generator().manual_seed(M)
    D = torch.randn(M, N, generator=g)
    D[::3] = 1.0                                                       # mantissa 0: -0.0 stays the pattern INT32_MIN
    any_bits = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, M + N), generator=g, dtype=torch.int64).to(torch.int32).view(torch.float32)
    any_bits = torch.where(any_bits.isfinite(), any_bits, torch.tensor(-0.0))
    any_bits[::4] = -0.0
    L, R = any_bits[:, :M].t().contiguous(), any_bits[:, M:].contiguous()
    if delta_l: L = torch.randn(M, K, generator=g)
    else: R = torch.randn(K, N, generator=g)
    want = oracle.kernels().pam_matmul_bwd(L, R, D, True, True, delta_l, 1.0)
    assert_bits_equal(cb._matmul_bwd(L.cuda(), R.cuda(), D.cuda(), delta_l, 1.0, 2, split_k=1), want)
