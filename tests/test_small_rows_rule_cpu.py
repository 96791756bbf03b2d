"""Which unsplit products take the tile of 56 rows, for either layout of A and width of the loads (no GPU needed)."""
import pytest

from pam_b200 import _lib


@pytest.mark.parametrize("batch,M,N,K,a_along_k,wide,rows", [
    (192, 197, 64, 197, 1, 0, 56), (192, 197, 64, 197, 0, 0, 56), (192, 197, 197, 64, 1, 0, 56),
    (500, 100, 100, 64, 1, 1, 56), (500, 100, 100, 64, 0, 0, 56),
    (500, 100, 100, 64, 0, 1, 64),                     # no such kernel for 128-bit loads along A's rows
    (192, 197, 197, 64, 1, 1, 32), (200, 151, 150, 150, 1, 0, 32),                  # dearer by the model
    (237, 146, 146, 128, 1, 0, 32), (394, 329, 90, 32, 0, 0, 32), (364, 65, 223, 128, 1, 0, 32),      # more than a fifth more outputs
    (1, 2400, 1460, 128, 1, 1, 64),
])
def test_rows_per_tile(batch, M, N, K, a_along_k, wide, rows):
    assert _lib.lib().pamk_test_small_rows(batch, M, N, K, a_along_k, wide) == rows


def test_empty_products_are_refused():
    assert _lib.lib().pamk_test_small_rows(1, 0, 4, 4, 1, 1) == -1
