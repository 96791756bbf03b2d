"""The 56x64 tile (seven rows per thread) and the walking scalar loads against the oracle, bit for bit: rows around multiples of 56 and of
the two groups of rows that a thread holds, columns around the tile's edge, K around slabs of 8, every layout and alignment,
a batch, a bias and lines of every kind."""
import pytest
import torch

from conftest import assert_bits_equal
from test_gpu_packed import _layout, _product
from test_gpu_special_lines import _values

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[5, 2, 3], ids=["tile56", "tile64", "tile32"])
def lib(request):
    from pam_b200 import _lib
    handle = _lib.lib()
    _lib.check(handle.pamk_test_set_tile_policy(request.param), "tile policy")
    handle.rows_per_tile = {5: 56, 2: 64, 3: 32}[request.param]
    yield handle
    handle.pamk_test_set_tile_policy(0)


def _takes_its_tile(lib, lay, batch, M, N, K):
    """The tile asked for is the one that runs, as all give the same bits: that of 56 rows has no kernel for 128-bit loads along A's
    rows (64 rows then)."""
    lone = {"n": K, "t": M}[lay[0].lower()] % 4 == 0 and {"n": N, "t": K}[lay[1].lower()] % 4 == 0 and lay.islower()
    a_along_k = lay[0] in "nN" or K == 1                  # (the operand's layout as the library sees it: a stride of 1 along K)
    want = 64 if lib.rows_per_tile == 56 and lone and not a_along_k else lib.rows_per_tile
    assert lib.pamk_test_small_rows(batch, M, N, K, a_along_k, lone) == want


@pytest.mark.parametrize("M", [1, 31, 32, 33, 55, 56, 57, 113])
@pytest.mark.parametrize("N,K", [(1, 1), (4, 4), (64, 8), (68, 20), (61, 17), (129, 40)])
@pytest.mark.parametrize("pool,share", [("none", 0.0), ("masked", 0.5), ("all", 0.02)])
def test_rows_and_loads(lib, M, N, K, pool, share, oracle):
    g = torch.Generator().manual_seed(M * 100 + N + K)
    A, B, bias = _values(pool, share, g, M, K), _values(pool, share, g, K, N), torch.randn(N, generator=g)
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, 1.0552) + bias
    for lay in ("nn", "nt", "tn", "tt", "Nt", "tN"):
        _takes_its_tile(lib, lay, 1, M, N, K)
        assert_bits_equal(_product(lib, _layout(A[None].cuda(), lay[0]), _layout(B[None].cuda(), lay[1]), bias=bias.cuda())[0], want, lay)


@pytest.mark.parametrize("batch,M,N,K", [(5, 197, 64, 197), (5, 64, 197, 197), (3, 100, 100, 64), (700, 57, 3, 9)])
def test_batches(lib, batch, M, N, K, oracle):
    g = torch.Generator().manual_seed(batch + M)
    A, B = _values("finite", 0.001, g, batch, M, K), _values("below", 0.001, g, batch, K, N)
    want = oracle.kernels().pam_bmm_fwd(A, B, True, True, 1.0552)
    for lay in ("nn", "tn", "Nt"):
        _takes_its_tile(lib, lay, batch, M, N, K)
        assert_bits_equal(_product(lib, _layout(A.cuda(), lay[0]), _layout(B.cuda(), lay[1])), want, lay)
