"""Large products under other allocators than torch's own, which answer no questions about their memory: they get their scratch like any
tensor, and their bits are the same."""
import os
import subprocess
import sys

import pytest
import torch

from conftest import ROOT, assert_bits_equal

pytestmark = pytest.mark.gpu

SIZE = 4096, 4096, 2048                                      # on packed operands: two passes over them and the product

CHILD = """
import sys, torch
if sys.argv[1]:
    allocator = torch.cuda.memory.CUDAPluggableAllocator(sys.argv[1], "plain_alloc", "plain_free")
    torch.cuda.memory.change_current_allocator(allocator)
import pam_b200 as pam
from pam_b200 import _lib, cuda_bindings as cb
pam.set_strict_k_order(True)
M, N, K = map(int, sys.argv[3:6])
A, B = (torch.linspace(-3, 5, n, device="cuda").view(shape) for n, shape in ((M * K, (M, K)), (K * N, (K, N))))
for product in (lambda: pam.matmul(A, B), lambda: cb._matmul(_lib.MUL_PAM, A, B, 1.0, 2)):
    launches = _lib.lib().pamk_launch_count()
    C = product()
    assert _lib.lib().pamk_launch_count() - launches == 3, "not on packed operands"
    torch.save(C.cpu(), sys.argv[2])
"""


@pytest.mark.parametrize("kind", ["pluggable", "cudaMallocAsync"])
def test_large_product(kind, tmp_path):
    import pam_b200 as pam
    plug = ""
    env = dict(os.environ, PYTHONPATH=str(ROOT))
    if kind == "pluggable":
        from pam_b200 import build
        plug = str(tmp_path / "libplain.so")
        subprocess.check_call([build._nvcc(), "-shared", "-Xcompiler", "-fPIC", "-o", plug, str(ROOT / "tests" / "plain_allocator.cpp")])
    else:
        env["PYTORCH_CUDA_ALLOC_CONF"] = "backend:cudaMallocAsync"
    out = tmp_path / "product.pt"
    M, N, K = SIZE
    done = subprocess.run([sys.executable, "-c", CHILD, plug, str(out), *map(str, SIZE)], env=env, cwd=ROOT, timeout=300, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr[-2000:]
    A, B = (torch.linspace(-3, 5, n, device="cuda").view(shape) for n, shape in ((M * K, (M, K)), (K * N, (K, N))))
    pam.set_strict_k_order(True)
    try:
        want = pam.matmul(A, B)
    finally:
        pam.set_strict_k_order(False)
    assert_bits_equal(torch.load(out).cuda(), want)
