"""Products in several K ranges on the 112x128 tile: the ranges and the order in which they are added are those of the 128x128 tile,
so every bit is the same, for rows and columns around the edges of both tiles, K around slabs, a bias and special values."""
import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 64, 67, 112, 113, 225, 4096])
@pytest.mark.parametrize("N,K,split", [(4, 64, 2), (132, 132, 3), (512, 512, 2), (60, 100, 7)])
def test_ranges_on_either_tile(M, N, K, split):
    from pam_b200 import _lib, cuda_bindings as cb
    lib = _lib.lib()
    g = torch.Generator().manual_seed(M + N + K)
    A, W, bias = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g), torch.randn(N, generator=g).cuda()
    pool = torch.tensor([0.0, 1e-40, 1e30, 1e-30, float("inf")])
    A[:, K // 3] = torch.where(torch.rand(M, generator=g) < 0.1, pool[torch.randint(0, 5, (M,), generator=g)], A[:, K // 3])
    A, W = A.cuda(), W.cuda()
    outs = []
    try:
        for policy, rows in ((1, 128), (4, 112)):
            _lib.check(lib.pamk_test_set_tile_policy(policy), "tile policy")
            assert lib.pamk_test_split_rows(M, N, K, split) == rows
            outs.append([cb._matmul(_lib.MUL_PAM, A, y, 1.0, 2, split_k=split, bias=b) for y in (W.t(), W.t().contiguous()) for b in (None, bias)])
    finally:
        lib.pamk_test_set_tile_policy(0)
    for have, want in zip(outs[1], outs[0]):
        assert_bits_equal(have, want)


def test_the_shapes_that_take_it():
    from pam_b200 import _lib
    lib = _lib.lib()
    for M, N, K, rows in ((4096, 512, 512, 112), (4096, 512, 1024, 128), (10000, 512, 4096, 128), (4096, 1024, 512, 112)):
        assert lib.pamk_test_split_rows(M, N, K, lib.pamk_matmul_auto_split(1, M, N, K)) == rows
