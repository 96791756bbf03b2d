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
STRADDLE = (1e-36, -1.1e-37, 9e-38, -3e-37)                                         # some products flush, none overflows
POOLS = {"masked": MASKED, "small": SMALL, "great": GREAT, "odd": ODD, "straddle": STRADDLE,
         "below": MASKED + SMALL + STRADDLE, "finite": MASKED + SMALL + STRADDLE + GREAT, "all": MASKED + SMALL + GREAT + ODD, "none": ()}


def _values(pool, share, g, *shape):
    t = torch.randn(*shape, generator=g)
    if POOLS[pool]:
        pick = torch.tensor(POOLS[pool])[torch.randint(0, len(POOLS[pool]), shape, generator=g)]
        t = torch.where(torch.rand(*shape, generator=g) < share, pick, t)
    return t


@pytest.mark.parametrize("policy", [1, 2, 3, 4], ids=["tile128", "tile64", "tile32", "tile112"])
@pytest.mark.parametrize("a_pool,b_pool", [("masked", "none"), ("none", "masked"), ("masked", "masked"), ("small", "none"),
                                           ("small", "small"), ("great", "none"), ("great", "masked"), ("masked", "great"),
                                           ("great", "small"), ("great", "great"), ("small", "masked"), ("odd", "none"),
                                           ("none", "odd"), ("straddle", "none"), ("straddle", "straddle"), ("straddle", "great"),
                                           ("all", "all")])
@pytest.mark.parametrize("share", [0.004, 0.3, 1.0])
@pytest.mark.parametrize("M,K,N", [(150, 53, 140), (148, 52, 140)], ids=["scalar loads", "128-bit loads"])
def test_lines_of_every_kind(policy, a_pool, b_pool, share, M, K, N, oracle):
    import pam_b200 as pam
    from pam_b200 import _lib
    from pam_b200.cuda_bindings import cuda_kernels
    offset = 1.0552
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


@pytest.mark.parametrize("policy", [1, 4], ids=["tile128", "tile112"])
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
def test_slabs_with_and_without_the_look(policy, layout, oracle):
    """90 slabs whose contents change so that looks are given up and taken up again: values around the flush bound, none, few dirty
    lines, every class on one side, the flush bound with elements above the band, few special values."""
    import pam_b200 as pam
    from pam_b200 import _lib
    from pam_b200.cuda_bindings import cuda_kernels
    M, K, N = 132, 1440, 136
    g = torch.Generator().manual_seed(7)
    A, B = torch.randn(M, K, generator=g), torch.randn(K, N, generator=g)
    A[:, :160] = _values("straddle", 1.0, g, M, 160)                   # looks are given up
    A[::9, 200:205], B[210, ::5] = 1e30, 1e-30                         # few dirty lines, with and without elements above the band
    A[:, 320:480], B[320:480] = _values("finite", 0.2, g, M, 160), _values("below", 0.2, g, 160, N)
    A[:, 640:800] = _values("straddle", 1.0, g, M, 160)
    B[700:760:3] = _values("great", 0.1, g, 20, N)                     # no look, elements above the band
    A[:, 1100:1300], B[1100:1300] = _values("finite", 0.01, g, M, 200), _values("below", 0.01, g, 200, N)     # looks again
    A[3, 730], B[1250, 7] = float("inf"), 3e38                         # NaN in one row and one column alone
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, 1.0)
    assert bool(want[3].isnan().all()) and bool(want[:, 7].isnan().any()) and float(want.isfinite().float().mean()) > 0.9
    x = A.cuda().t().contiguous().t() if layout[0] == "t" else A.cuda()
    y = B.cuda().t().contiguous().t() if layout[1] == "t" else B.cuda()
    _lib.check(_lib.lib().pamk_test_set_tile_policy(policy), "tile policy")
    pam.set_strict_k_order(True)
    try:
        assert_bits_equal(cuda_kernels.pam_matmul_fwd(x, y, True, True, 1.0), want)
    finally:
        pam.set_strict_k_order(False)
        _lib.lib().pamk_test_set_tile_policy(0)
