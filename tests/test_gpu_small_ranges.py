"""Small products in ranges of K that run in one launch: each range summed in k order and the ranges added in theirs, which the oracle
does range by range; rows, columns and K around the edges of tiles and slabs, every layout and alignment, a batch, a bias, a
strided output with a PAM multiplication, special values."""
import pytest
import torch

from conftest import assert_bits_equal
from test_gpu_packed import _layout, _product
from test_gpu_special_lines import _values

pytestmark = pytest.mark.gpu


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
        assert_bits_equal(_product(lib, _layout(A.cuda(), lay[0]), _layout(B.cuda(), lay[1]), split, bias.cuda()), want, lay)


def test_a_batch_and_a_strided_output(lib, oracle):
    from pam_b200 import _lib
    batch, M, N, K, split, ld = 3, 20, 37, 130, 3, 41
    g = torch.Generator().manual_seed(2)
    A, B = _values("all", 0.01, g, batch, M, K), _values("below", 0.01, g, batch, K, N)
    want = _in_ranges(oracle, A, B, split, 1.0)
    assert_bits_equal(_product(lib, A.cuda(), B.cuda(), split, offset=1.0), want)
    out, x, y = torch.full((batch, M, ld), -7.0, device="cuda"), A.cuda(), B.cuda()
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
