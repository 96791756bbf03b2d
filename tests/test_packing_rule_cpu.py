"""Which products run on packed operands, from the scratch that they ask for (no GPU needed)."""
import pytest

from pam_b200 import _lib


@pytest.mark.parametrize("M,N,K,packs", [
    (4096, 4096, 4096, True), (8192, 8192, 8192, True), (4096, 10000, 512, True), (6000, 3000, 2000, True), (2048, 2048, 2048, False), (4096, 4096, 512, False),
    (10000, 512, 4096, False), (4096, 512, 512, False), (4096, 1024, 512, False),      # too few columns: the passes cost what they save
    (4096, 2048, 512, False), (1024, 512, 4096, False), (16384, 256, 16384, False),
])
def test_large_products_in_both_dimensions_are_packed(M, N, K, packs):
    lib = _lib.lib()
    for split in (0, 1, 2):
        planned = split or lib.pamk_matmul_auto_split(1, M, N, K)
        partials = (lib.pamk_matmul_workspace_bytes(1, M, N, planned) + 255) // 256 * 256
        scratch = lib.pamk_matmul_scratch_bytes(1, M, N, K, split)
        # 16 x 128 floats and 336 bytes of masks and flags for each block of either operand, and the extremes of each line
        tile = 128 if not packs or lib.pamk_test_split_rows(M, N, K, split) == 128 else 112
        blocks = (-(-M // tile) + -(-N // 128)) * -(-K // 16)
        extremes = 2 * (-(-(-(-K // 16) * 16 * 8) // 256) * 256)
        large = lib.pamk_test_planned_rows(M, N, K, split) >= 112        # (some splits go to a smaller tile)
        assert large or split != 0
        assert scratch == partials + (extremes + blocks * (16 * 128 * 4 + 336) if packs and large else 0)


def test_products_below_the_stated_size_take_no_more():
    lib = _lib.lib()
    for shape in ((1, 1442, 1442, 1442), (64, 360, 360, 360), (1, 16384, 16384, 11), (1, 2080, 60000, 24)):
        assert shape[0] * shape[1] * shape[2] * shape[3] <= 3e9
        assert lib.pamk_matmul_scratch_bytes(*shape, 1) == 0
    assert lib.pamk_matmul_scratch_bytes(1, 0, 5, 5, 0) == 0 and lib.pamk_matmul_scratch_bytes(1, 5, 5, 5, -1) == 0
