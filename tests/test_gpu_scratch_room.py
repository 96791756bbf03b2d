"""Large products where torch's allocator has no room for their packed operands: they run on the operands as they are, with the same
bits, and what the allocator has cached stays where it is."""
import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("native", [True, False])
def test_no_room(native):
    import pam_b200 as pam
    from pam_b200 import _lib, cuda_bindings as cb
    lib = _lib.lib()
    M, N, K = 4096, 4096, 2048
    torch.cuda.empty_cache()
    pam.set_strict_k_order(True)                             # (one range: no partial sums, which a product cannot do without)
    A, B = torch.randn(M, K, device="cuda"), torch.randn(K, N, device="cuda")
    product = (lambda: pam.matmul(A, B)) if native else (lambda: cb._matmul(_lib.MUL_PAM, A, B, 1.0, 2))
    launches = lib.pamk_launch_count()
    want = product()
    packed = lib.pamk_launch_count() - launches
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cached = [torch.empty(64 << 20, dtype=torch.uint8, device="cuda") for _ in range(4)]        # room for results, not for scratch
    del cached
    total, before = torch.cuda.mem_get_info()[1], torch.cuda.get_per_process_memory_fraction()
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (32 << 20)) / total)
        stats = torch.cuda.memory_stats()
        launches = lib.pamk_launch_count()
        have = [product() for _ in range(3)]
        in_place = lib.pamk_launch_count() - launches
        after = torch.cuda.memory_stats()
    finally:
        torch.cuda.set_per_process_memory_fraction(before)
        pam.set_strict_k_order(False)
    for h in have:
        assert_bits_equal(h, want)
    assert packed == 3 and in_place == 3                     # (pack, classify, product; three products)
    for key in ("num_ooms", "num_alloc_retries"):
        assert after[key] == stats[key], key
    assert after["reserved_bytes.all.current"] == stats["reserved_bytes.all.current"]
