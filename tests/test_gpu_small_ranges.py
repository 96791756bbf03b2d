"""Small products in ranges of K that run in one launch: each range summed in k order and the ranges added in theirs, which the oracle
does range by range; rows, columns and K around the edges of tiles and slabs, every layout and alignment, a batch, a bias, a
strided output with a PAM multiplication, special values."""
import contextlib

import pytest
import torch

from conftest import assert_bits_equal
from test_gpu_packed import _layout, _product
from test_gpu_special_lines import GREAT, MASKED, ODD, SMALL, STRADDLE, _values

pytestmark = pytest.mark.gpu

ZEROS = (0.0, -0.0)


@contextlib.contextmanager
def _launches(lib, count):
    """The kernels launched inside are this many: which form a product took, as all forms give the same bits."""
    before = lib.pamk_launch_count()
    yield
    assert lib.pamk_launch_count() - before == count


@pytest.fixture
def lib():
    from pam_b200 import _lib
    handle = _lib.lib()
    _lib.check(handle.pamk_test_set_tile_policy(3), "tile policy")
    yield handle
    handle.pamk_test_set_tile_policy(0)


def _in_ranges(oracle, A, B, split, offset):
    """The oracle's products of the ranges that the library cuts K into (whole slabs of 16), added in order."""
    slabs = -(-A.shape[-1] // 16)
    chunk = -(-slabs // split) * 16
    total = None
    for k in range(0, A.shape[-1], chunk):
        part = oracle.kernels().pam_bmm_fwd(A[..., k:k + chunk].contiguous(), B[..., k:k + chunk, :].contiguous(), True, True, offset)
        total = part if total is None else total + part
    return total


@pytest.mark.parametrize("M,N", [(1, 1), (1, 500), (15, 17), (16, 16), (32, 64), (33, 47), (100, 130)])
@pytest.mark.parametrize("K,split", [(17, 2), (32, 2), (96, 3), (100, 4), (250, 16), (512, 16), (517, 7)])
@pytest.mark.parametrize("pool,share", [("none", 0.0), ("all", 0.01)])
def test_ranges_in_one_launch(lib, M, N, K, split, pool, share, oracle):
    g = torch.Generator().manual_seed(M * 31 + N + K)
    A, B, bias = _values(pool, share, g, 1, M, K), _values(pool, share, g, 1, K, N), torch.randn(N, generator=g)
    want = _in_ranges(oracle, A, B, split, 1.0552) + bias
    for lay in ("nn", "nt", "tn", "Tt"):
        x, y, b = _layout(A.cuda(), lay[0]), _layout(B.cuda(), lay[1]), bias.cuda()
        with _launches(lib, 1 if K < 517 else 2):             # (517 in 7: ranges of five slabs are too long for one launch)
            have = _product(lib, x, y, split, b)
        assert_bits_equal(have, want, lay)


@pytest.mark.parametrize("M,N,K,split", [(33, 47, 100, 4), (20, 300, 50, 3), (208, 192, 512, 16)])
@pytest.mark.parametrize("a_pool,b_pool,share", [(ZEROS, (), 0.5), ((), ZEROS, 0.5), (ZEROS, ZEROS, 0.3), (ZEROS, ZEROS, 0.01), (STRADDLE, (), 0.01),
                                                 (SMALL, STRADDLE, 0.3), (GREAT, MASKED, 0.01), (ODD, GREAT, 0.01), (GREAT, ODD, 0.3)])
def test_slabs_of_every_kind(lib, M, N, K, split, a_pool, b_pool, share, oracle):
    """Each loop for dirty slabs, in all slabs and in some of them: a warp's two ranges see different kinds, and the last may be alone."""
    g = torch.Generator().manual_seed(M + len(a_pool) * 10 + int(share * 1000))
    def values(pool, *shape):
        t = torch.randn(*shape, generator=g)
        if pool:
            pick = torch.tensor(pool)[torch.randint(0, len(pool), shape, generator=g)]
            t = torch.where(torch.rand(*shape, generator=g) < share, pick, t)
        return t
    A, B = values(a_pool, 1, M, K), values(b_pool, 1, K, N)
    for some in (False, True):
        if some:                                             # every third slab as it is, the others clean
            clean = (torch.arange(K) // 16 % 3 != 0)
            A[..., clean], B[:, clean] = torch.randn(1, M, int(clean.sum()), generator=g), torch.randn(1, int(clean.sum()), N, generator=g)
        want = _in_ranges(oracle, A, B, split, 1.0552)
        for lay in ("nn", "nt", "tn", "Nt"):
            x, y = _layout(A.cuda(), lay[0]), _layout(B.cuda(), lay[1])
            with _launches(lib, 1):
                have = _product(lib, x, y, split)
            assert_bits_equal(have, want, lay)


def test_a_batch_and_a_strided_output(lib, oracle):
    from pam_b200 import _lib
    batch, M, N, K, split, ld = 3, 20, 37, 130, 3, 41
    g = torch.Generator().manual_seed(2)
    A, B = _values("all", 0.01, g, batch, M, K), _values("below", 0.01, g, batch, K, N)
    want = _in_ranges(oracle, A, B, split, 1.0)
    x, y = A.cuda(), B.cuda()
    with _launches(lib, 1):
        have = _product(lib, x, y, split, offset=1.0)
    assert_bits_equal(have, want)
    out = torch.full((batch, M, ld), -7.0, device="cuda")
    ws = torch.empty(split * batch * M * N, device="cuda")
    _lib.check(lib.pamk_matmul_strided(x.data_ptr(), y.data_ptr(), out.data_ptr(), 1, batch, M, N, K, 0, M * K, K, 1, 0, K * N, N, 1, 0, M * ld, ld,
                                       1.0, 1, 0.125, split, ws.data_ptr(), 4 * ws.numel(), torch.cuda.current_stream().cuda_stream), "strided")
    assert_bits_equal(out[..., :N], oracle.kernels().pam_fwd(want.contiguous(), torch.full_like(want, 0.125), 1.0))
    assert bool((out[..., N:] == -7.0).all())


def test_scratch_is_asked_for_as_before(lib):
    """An explicit split without scratch is refused, and the library's choice without scratch is one range."""
    x, out = torch.randn(32, 512, device="cuda"), torch.empty(32, 32, device="cuda")
    for split, status in ((16, -4), (0, 0)):
        assert lib.pamk_matmul(0, x.data_ptr(), x.data_ptr(), out.data_ptr(), 1, 32, 32, 512, 0, 512, 1, 0, 1, 512, 1.0, split, None, 0,
                               torch.cuda.current_stream().cuda_stream) == status
