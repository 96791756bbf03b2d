"""The 112x128 tile (seven rows per thread) against the oracle, bit for bit: rows around multiples of 112 and of the two
groups of rows that a thread holds, columns around the tile's edge, K around slabs, both layouts of B, a bias, and values
outside the band in every row slot.  Unsplit sums are in the reference's order whatever the tile."""
import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.fixture
def seven_rows():
    import pam_b200 as pam
    from pam_b200 import _lib
    _lib.check(_lib.lib().pamk_test_set_tile_policy(4), "tile policy")
    pam.set_strict_k_order(True)
    yield
    pam.set_strict_k_order(False)
    _lib.lib().pamk_test_set_tile_policy(0)


@pytest.mark.parametrize("M", [1, 63, 64, 65, 67, 111, 112, 113, 225])
@pytest.mark.parametrize("N,K", [(4, 4), (128, 16), (132, 36), (60, 100)])
@pytest.mark.parametrize("special", [0.0, 0.02])
def test_seven_rows_per_thread(seven_rows, M, N, K, special, oracle):
    from pam_b200 import _lib, cuda_bindings as cb
    g = torch.Generator().manual_seed(M * 100 + N + K)
    A, B, bias = torch.randn(M, K, generator=g), torch.randn(K, N, generator=g), torch.randn(N, generator=g)
    for t in (A, B):
        pool = torch.tensor([0.0, 1e-40, 1e30, 1e-30, float("inf")])
        pick = pool[torch.randint(0, 5, t.shape, generator=g)]
        t.copy_(torch.where(torch.rand(t.shape, generator=g) < special, pick, t))
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, 1.0)
    for y in (B.cuda(), B.cuda().t().contiguous().t()):
        assert_bits_equal(cb._matmul(_lib.MUL_PAM, A.cuda(), y, 1.0, 2), want)
        assert_bits_equal(cb._matmul(_lib.MUL_PAM, A.cuda(), y, 1.0, 2, bias=bias.cuda()), want + bias)


def test_the_planner_takes_it_where_it_fits_the_sms(oracle):
    """4096x512 in tiles of 112 rows is one per SM: the automatic product is not split and keeps the reference's order."""
    from pam_b200 import _lib, cuda_bindings as cb
    g = torch.Generator().manual_seed(5)
    A, W = torch.randn(4096, 512, generator=g).cuda(), torch.randn(512, 512, generator=g).cuda()
    got = cb._matmul(_lib.MUL_PAM, A, W.t(), 1.0, 2)
    assert torch.equal(got, cb._matmul(_lib.MUL_PAM, A, W.t(), 1.0, 2, split_k=1))
    assert torch.equal(got[:3].cpu(), oracle.kernels().pam_matmul_fwd(A[:3].cpu(), W.t().cpu(), True, True, 1.0))
