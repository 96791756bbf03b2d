"""Products whose k lines mix values of every magnitude class: zeros and denormals, small and great values that pass with
ordinary partners, inf and NaN, alone and beside one another on either side, against the oracle, bit for bit.  Each warp
chooses a loop per line from what its own rows and columns hold, so the values are placed sparsely (most warps
see one kind) and densely (most see several)."""
import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu

MASKED = (0.0, -0.0, 1e-40, -1.4e-45, 3e-38)
SMALL = (1e-30, -1e-25, 3e-20)
GREAT = (1e30, -1e25, 1e19)
ODD = (float("inf"), float("-inf"), float("nan"), 3e38, -2e37, 1e-36, 1.1e-37)      # the last ones flush with some partners
POOLS = {"masked": MASKED, "small": SMALL, "great": GREAT, "odd": ODD, "all": MASKED + SMALL + GREAT + ODD, "none": ()}


def _values(pool, share, g, *shape):
    t = torch.randn(*shape, generator=g)
    if POOLS[pool]:
        pick = torch.tensor(POOLS[pool])[torch.randint(0, len(POOLS[pool]), shape, generator=g)]
        t = torch.where(torch.rand(*shape, generator=g) < share, pick, t)
    return t


@pytest.mark.parametrize("policy", [1, 2, 3], ids=["tile128", "tile64", "tile32"])
@pytest.mark.parametrize("a_pool,b_pool", [("masked", "none"), ("none", "masked"), ("masked", "masked"), ("small", "none"),
                                           ("small", "small"), ("great", "none"), ("great", "masked"), ("masked", "great"),
                                           ("great", "small"), ("great", "great"), ("small", "masked"), ("odd", "none"),
                                           ("none", "odd"), ("all", "all")])
@pytest.mark.parametrize("share", [0.004, 0.3, 1.0])
def test_lines_of_every_kind(policy, a_pool, b_pool, share, oracle):
    import pam_b200 as pam
    from pam_b200 import _lib
    from pam_b200.cuda_bindings import cuda_kernels
    M, K, N, offset = 150, 53, 140, 1.0552
    g = torch.Generator().manual_seed(len(a_pool) * 100 + len(b_pool) + int(share * 1000))
    A, B = _values(a_pool, share, g, M, K), _values(b_pool, share, g, K, N)
    A[5], B[:, 7] = 0.0, 0.0                       # one row and one column that are masked in every line
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, offset)
    _lib.check(_lib.lib().pamk_test_set_tile_policy(policy), "tile policy")
    pam.set_strict_k_order(True)
    try:
        for x in (A.cuda(), A.cuda().t().contiguous().t()):
            for y in (B.cuda(), B.cuda().t().contiguous().t()):
                assert_bits_equal(cuda_kernels.pam_matmul_fwd(x, y, True, True, offset), want)
    finally:
        pam.set_strict_k_order(False)
        _lib.lib().pamk_test_set_tile_policy(0)
