"""The 112x128 tile (seven rows per thread) against the oracle, bit for bit: rows around multiples of 112 and of the two
groups of rows that a thread holds, columns around the tile's edge, K around slabs, both layouts of B, a bias, and values
outside the band in every row slot.  Unsplit sums are in the reference's order whatever the tile; a product that the
plan of its shape cuts along K does not take this tile."""
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
    assert _lib.lib().pamk_test_planned_rows(M, N, K, 1) == 112
    for t in (A, B):
        pool = torch.tensor([0.0, 1e-40, 1e30, 1e-30, float("inf")])
        pick = pool[torch.randint(0, 5, t.shape, generator=g)]
        t.copy_(torch.where(torch.rand(t.shape, generator=g) < special, pick, t))
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, 1.0)
    for y in (B.cuda(), B.cuda().t().contiguous().t()):
        assert_bits_equal(cb._matmul(_lib.MUL_PAM, A.cuda(), y, 1.0, 2), want)
        assert_bits_equal(cb._matmul(_lib.MUL_PAM, A.cuda(), y, 1.0, 2, bias=bias.cuda()), want + bias)


def _specials(t, g, share=0.02):
    pool = torch.tensor([0.0, 1e-40, 1e30, 1e-30, float("inf")])
    return torch.where(torch.rand(t.shape, generator=g) < share, pool[torch.randint(0, 5, t.shape, generator=g)], t)


def _policy(policy):
    from pam_b200 import _lib
    _lib.check(_lib.lib().pamk_test_set_tile_policy(policy), "tile policy")


def _off_by_one(t):
    """The same values one float further: 4-byte aligned storage."""
    buf = torch.empty(t.numel() + 1, device=t.device)
    return buf[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("M,N,K", [(4096, 512, 512), (4104, 512, 1024), (1000, 2048, 512), (2304, 768, 256), (3000, 2048, 1024)])
def test_the_order_of_the_sums_follows_from_the_shape_alone(M, N, K):
    """Shapes that the planner cuts along K and that would run faster unsplit on this tile where A lies contiguous along K and
    aligned: those, a transposed operand and one that starts a float further all have to add the same ranges in the same order."""
    from pam_b200 import _lib, cuda_bindings as cb
    lib = _lib.lib()
    split = lib.pamk_matmul_auto_split(1, M, N, K)
    assert split > 1 and lib.pamk_test_planned_rows(M, N, K, split) != 112
    g = torch.Generator().manual_seed(M + K)
    A, W, bias = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g), torch.randn(N, generator=g).cuda()
    A[:, K // 3] = _specials(A[:, K // 3], g)
    A, W = A.cuda(), W.cuda()
    for b in (None, bias):
        want = cb._matmul(_lib.MUL_PAM, A.t().contiguous().t(), W.t(), 1.0, 2, bias=b)
        for x, y in ((A, W.t()), (A, W.t().contiguous()), (_off_by_one(A), W.t()), (A, _off_by_one(W).t())):
            assert_bits_equal(cb._matmul(_lib.MUL_PAM, x, y, 1.0, 2, bias=b), want)
    # (a split of one range is another order: the comparison above could not pass by chance)
    one = cb._matmul(_lib.MUL_PAM, A, W.t(), 1.0, 2, split_k=1, bias=bias)
    assert not torch.equal(want.nan_to_num(nan=0.0), one.nan_to_num(nan=0.0))


def test_operands_that_the_tile_does_not_take(seven_rows, oracle):
    """Where the tile is asked for and the operands do not allow it: A contiguous along its rows, storage that is not 16-byte
    aligned, K no multiple of 4, a batch."""
    from pam_b200 import _lib, cuda_bindings as cb
    g = torch.Generator().manual_seed(3)
    for M, N, K in ((230, 132, 64), (225, 60, 37)):
        A, B = _specials(torch.randn(M, K, generator=g), g), _specials(torch.randn(K, N, generator=g), g)
        want = oracle.kernels().pam_matmul_fwd(A, B, True, True, 1.0)
        for x in (A.cuda(), A.cuda().t().contiguous().t(), _off_by_one(A.cuda())):
            for y in (B.cuda(), B.cuda().t().contiguous().t(), _off_by_one(B.cuda())):
                assert_bits_equal(cb._matmul(_lib.MUL_PAM, x, y, 1.0, 2), want)
    A, B = _specials(torch.randn(3, 120, 64, generator=g), g), _specials(torch.randn(3, 64, 36, generator=g), g)
    assert_bits_equal(cb._matmul(_lib.MUL_PAM, A.cuda(), B.cuda(), 1.0, 3), oracle.kernels().pam_bmm_fwd(A, B, True, True, 1.0))


@pytest.mark.parametrize("split", [1, 3])
def test_strided_output_between_canaries(split):
    """One matrix of pamk_matmul_strided with rows further apart than they are long and a PAM multiplication of the sums: the
    gaps stay as they were."""
    from pam_b200 import _lib
    g = torch.Generator().manual_seed(4)
    M, N, K, ld = 230, 60, 256, 68
    A, W = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    ws = torch.empty(split * M * N, device="cuda")
    outs = []
    try:
        for policy in (1, 4):
            _policy(policy)
            buf = torch.full((64 + M * ld + 64,), -7.0, device="cuda")
            _lib.check(_lib.lib().pamk_matmul_strided(A.data_ptr(), W.data_ptr(), buf[64:].data_ptr(), 1, 1, M, N, K, 0, 0, K, 1, 0, 0, 1, K,
                                                      0, 0, ld, 1.0552, 1, 0.125, split, ws.data_ptr(), 4 * ws.numel(),
                                                      torch.cuda.current_stream().cuda_stream), "strided")
            outs.append(buf)
    finally:
        _policy(0)
    assert_bits_equal(outs[1], outs[0])
    rows = outs[1][64:64 + M * ld].view(M, ld)
    assert bool((rows[:, N:] == -7.0).all()) and bool((outs[1][:64] == -7.0).all()) and bool((outs[1][64 + M * ld:] == -7.0).all())
    assert not bool((rows[:, :N] == -7.0).any())


def test_too_little_scratch(oracle):
    """The library's choice without scratch is one range; an explicit split without it is refused, whatever the tile."""
    from pam_b200 import _lib, cuda_bindings as cb
    g = torch.Generator().manual_seed(5)
    M, N, K = 4096, 512, 512
    A, W = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    out = torch.full((M, N), -7.0, device="cuda")
    ws = torch.empty(1024, dtype=torch.uint8, device="cuda")
    for split, status in ((0, 0), (2, -4)):
        for p, n in ((None, 0), (ws.data_ptr(), ws.numel())):
            assert _lib.lib().pamk_matmul(0, A.data_ptr(), W.data_ptr(), out.data_ptr(), 1, M, N, K, 0, K, 1, 0, 1, K, 1.0, split, p, n,
                                          torch.cuda.current_stream().cuda_stream) == status
    assert_bits_equal(out, cb._matmul(_lib.MUL_PAM, A, W.t(), 1.0, 2, split_k=1))
    assert_bits_equal(out[:3].cpu(), oracle.kernels().pam_matmul_fwd(A[:3].cpu(), W.t().cpu(), True, True, 1.0))
