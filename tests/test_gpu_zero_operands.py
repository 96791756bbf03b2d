"""Products whose operands hold zeros and otherwise only values of ordinary magnitude (an operand that went through
a ReLU), against the oracle, bit for bit: a slab whose out-of-band elements are all zeros takes a loop of its own,
one that also holds other elements, or few zeros, does not.
"""
import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


def _with_zeros(share, g, *shape):
    t = torch.randn(*shape, generator=g)
    zero = torch.rand(*shape, generator=g) < share
    sign = torch.where(torch.rand(*shape, generator=g) < 0.5, 0.0, -0.0)
    return torch.where(zero, sign, t)


@pytest.mark.parametrize("policy", [1, 2, 3], ids=["tile128", "tile64", "tile32"])
@pytest.mark.parametrize("M,K,N", [(1, 8, 1), (33, 16, 65), (128, 40, 128), (130, 197, 67), (64, 64, 260)])
@pytest.mark.parametrize("a_share,b_share", [(0.5, 0.0), (0.0, 0.5), (0.5, 0.5), (1.0, 0.0), (0.0, 1.0), (0.01, 0.01)])
@pytest.mark.parametrize("offset", [1.0, 0.97, 1.0552])
def test_zeros_in_an_operand(policy, M, K, N, a_share, b_share, offset, oracle):
    import pam_b200 as pam
    from pam_b200 import _lib
    from pam_b200.cuda_bindings import cuda_kernels
    g = torch.Generator().manual_seed(M * 1000 + K + N)
    A, B = _with_zeros(a_share, g, M, K), _with_zeros(b_share, g, K, N)
    mixed = A.clone()
    mixed[M // 2, K // 2] = 1e-30                 # one slab holds another out-of-band element beside its zeros
    _lib.check(_lib.lib().pamk_test_set_tile_policy(policy), "tile policy")
    pam.set_strict_k_order(True)
    try:
        for a in (A, mixed):
            want = oracle.kernels().pam_matmul_fwd(a, B, True, True, offset)
            for a_t in (False, True):
                for b_t in (False, True):
                    x = a.cuda().t().contiguous().t() if a_t else a.cuda()
                    y = B.cuda().t().contiguous().t() if b_t else B.cuda()
                    assert_bits_equal(cuda_kernels.pam_matmul_fwd(x, y, not a_t, not b_t, offset), want, f"layouts {a_t} {b_t}")
    finally:
        pam.set_strict_k_order(False)
        _lib.lib().pamk_test_set_tile_policy(0)


@pytest.mark.parametrize("policy", [1, 2, 3], ids=["tile128", "tile64", "tile32"])
@pytest.mark.parametrize("every", [1, 3, 12])
def test_slabs_of_zeros_among_slabs_that_hold_others(policy, every, oracle):
    """Slabs whose many out-of-band elements are all zeros among slabs where they are not: runs of both sorts, of several
    lengths (K is 40 slabs of 16)."""
    import pam_b200 as pam
    from pam_b200 import _lib
    from pam_b200.cuda_bindings import cuda_kernels
    g = torch.Generator().manual_seed(every)
    M, K, N = 70, 640, 65
    A, B = _with_zeros(0.5, g, M, K), _with_zeros(0.0, g, K, N)
    for first in range(0, K, 16 * every):
        A[::3, first:first + 16] *= 2.0 ** -64                   # below the band
    B[::7, :] = torch.where(torch.rand(B[::7].shape, generator=g) < 0.5, 0.0, B[::7])
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, 1.0)
    _lib.check(_lib.lib().pamk_test_set_tile_policy(policy), "tile policy")
    pam.set_strict_k_order(True)
    try:
        for x in (A.cuda(), A.cuda().t().contiguous().t()):
            for y in (B.cuda(), B.cuda().t().contiguous().t()):
                assert_bits_equal(cuda_kernels.pam_matmul_fwd(x, y, True, True, 1.0), want)
    finally:
        pam.set_strict_k_order(False)
        _lib.lib().pamk_test_set_tile_policy(0)


@pytest.mark.parametrize("K", [5, 8, 17, 24, 21])
@pytest.mark.parametrize("share", [(0.5, 0.0), (0.0, 0.5), (0.5, 0.5), (0.0, 0.0)])
def test_many_small_products_whose_k_ends_early_in_a_slab(K, share, oracle):
    """More than four 32x32 tiles per SM and K just past a multiple of 16: the slabs of 8 of that tile, on zeros and on
    other out-of-band values."""
    import pam_b200 as pam
    from pam_b200 import _lib
    from pam_b200.cuda_bindings import cuda_kernels
    g = torch.Generator().manual_seed(K)
    batch, M, N = 1300, 30, 31
    A, B = _with_zeros(share[0], g, batch, M, K), _with_zeros(share[1], g, batch, K, N)
    A.view(-1)[::997], B.view(-1)[::1009] = 1e-30, 1e30
    want = oracle.kernels().pam_bmm_fwd(A, B, True, True, 1.0552)
    _lib.check(_lib.lib().pamk_test_set_tile_policy(3), "tile policy")
    pam.set_strict_k_order(True)
    try:
        for x in (A.cuda(), A.cuda().mT.contiguous().mT):
            for y in (B.cuda(), B.cuda().mT.contiguous().mT):
                assert_bits_equal(cuda_kernels.pam_bmm_fwd(x, y, True, True, 1.0552), want)
    finally:
        pam.set_strict_k_order(False)
        _lib.lib().pamk_test_set_tile_policy(0)
