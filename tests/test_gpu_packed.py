"""PAM products on packed operands: against the oracle bit for bit where one range is summed, and against the same product on the
operands as they are for everything else.  Sizes around the edges of tiles (128 or 112 rows), slabs (16 k), the passes' groups (64 k) and
the ring (6 slabs), every layout and alignment of the operands, batches, ranges of K, a bias, strided outputs, and lines of
every kind."""
import ctypes

import pytest
import torch

from conftest import assert_bits_equal
from test_gpu_special_lines import _values

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 4], ids=["tile128", "tile112"])
def packed(request):
    from pam_b200 import _lib
    lib = _lib.lib()
    _lib.check(lib.pamk_test_set_tile_policy(request.param), "tile policy")
    _lib.check(lib.pamk_test_set_packing_policy(1), "packing")
    yield lib
    count = ctypes.c_uint(7)
    lib.pamk_test_set_tile_policy(0)
    lib.pamk_test_set_packing_policy(0)
    _lib.check(lib.pamk_test_expired_waits(ctypes.byref(count)), "expired waits")
    assert count.value == 0


def _layout(t, kind):
    """The same matrix: row-major, column-major, or either one float past a 16-byte boundary."""
    rows_first = t if kind in ("n", "N") else t.transpose(-1, -2)
    buf = torch.empty(t.numel() + 1, device="cuda")
    at = buf[1:] if kind.isupper() else buf[:-1]
    view = at.view(rows_first.shape).copy_(rows_first)
    return view if kind in ("n", "N") else view.transpose(-1, -2)


def _product(lib, x, y, split=1, bias=None, offset=1.0552, scratch=None, launches=None):
    from pam_b200 import _lib
    batch, (M, K), N = x.shape[0], x.shape[1:], y.shape[2]
    nbytes = lib.pamk_matmul_scratch_bytes(batch, M, N, K, split)
    ws = torch.full((max(nbytes if scratch is None else scratch, 1),), 0x5a, dtype=torch.uint8, device="cuda")
    out = torch.full((batch, M, N), -7.0, device="cuda")
    before = lib.pamk_launch_count()
    _lib.check(lib.pamk_matmul_bias(0, x.data_ptr(), y.data_ptr(), None if bias is None else bias.data_ptr(), out.data_ptr(), batch, M, N, K,
                                    *x.stride(), *y.stride(), offset, split, ws.data_ptr(), ws.numel(),
                                    torch.cuda.current_stream().cuda_stream), "product")
    # (which form it took, as all forms give the same bits: three launches on packed operands, one in place, and the sum of the ranges)
    assert launches is None or lib.pamk_launch_count() - before == launches + (1 if split > 1 else 0)
    return out


def _in_place(lib, *args, **kw):
    lib.pamk_test_set_packing_policy(2)
    try:
        return _product(lib, *args, launches=1, **kw)
    finally:
        lib.pamk_test_set_packing_policy(1)


@pytest.mark.parametrize("a_pool,b_pool,share", [("none", "none", 0.0), ("masked", "none", 0.5), ("none", "masked", 0.01), ("masked", "masked", 0.3),
                                                 ("great", "masked", 0.01), ("small", "small", 0.02), ("great", "great", 0.004), ("straddle", "great", 0.3),
                                                 ("odd", "none", 0.004), ("none", "odd", 0.004), ("all", "all", 0.02), ("all", "all", 1.0)])
@pytest.mark.parametrize("M,K,N", [(150, 53, 140), (148, 52, 140), (113, 200, 129)])
def test_lines_of_every_kind(packed, a_pool, b_pool, share, M, K, N, oracle):
    g = torch.Generator().manual_seed(M + len(a_pool) * 100 + len(b_pool) + int(share * 1000))
    A, B = _values(a_pool, share, g, M, K), _values(b_pool, share, g, K, N)
    if a_pool != "none": A[5] = 0.0
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, 1.0552)
    for lay in ("nn", "nt", "tn", "tt", "Nt", "tN"):
        assert_bits_equal(_product(packed, _layout(A[None].cuda(), lay[0]), _layout(B[None].cuda(), lay[1]), launches=3)[0], want, lay)


@pytest.mark.parametrize("M,N", [(1, 1), (1, 300), (64, 64), (67, 127), (112, 128), (113, 129), (225, 4), (260, 256)])
@pytest.mark.parametrize("K", [1, 15, 16, 17, 63, 64, 65, 96, 97, 112, 130])
def test_edges(packed, M, N, K, oracle):
    g = torch.Generator().manual_seed(M * 7 + N + K)
    A, B, bias = _values("all", 0.002, g, M, K), _values("all", 0.002, g, K, N), torch.randn(N, generator=g)
    want = oracle.kernels().pam_matmul_fwd(A, B, True, True, 1.0552) + bias
    for lay in ("nt", "tn"):
        assert_bits_equal(_product(packed, _layout(A[None].cuda(), lay[0]), _layout(B[None].cuda(), lay[1]), bias=bias.cuda(), launches=3)[0], want, lay)


@pytest.mark.parametrize("batch,M,N,K,split", [(3, 130, 70, 100, 1), (2, 113, 132, 200, 3), (1, 300, 260, 1000, 5), (1, 260, 512, 2000, 1)])
def test_batches_ranges_and_scratch(packed, batch, M, N, K, split):
    g = torch.Generator().manual_seed(M + K)
    A, B, bias = _values("finite", 0.003, g, batch, M, K), _values("below", 0.003, g, batch, K, N), torch.randn(N, generator=g).cuda()
    for lay in ("nn", "nt", "tn", "Tt"):
        x, y = _layout(A.cuda(), lay[0]), _layout(B.cuda(), lay[1])
        want = _in_place(packed, x, y, split, bias)
        assert_bits_equal(_product(packed, x, y, split, bias, launches=3), want, lay)
        # one byte too little for the packed operands: the product runs on them as they are
        assert_bits_equal(_product(packed, x, y, split, bias, scratch=packed.pamk_matmul_scratch_bytes(batch, M, N, K, split) - 1,
                                   launches=1), want, lay)


def test_heads_of_a_fused_projection(packed):
    """pamk_matmul_strided: a two-level batch, an output between canaries, a PAM multiplication of the finished sums."""
    from pam_b200 import _lib
    outer, heads, M, N, K, ld = 2, 3, 130, 68, 100, 72
    g = torch.Generator().manual_seed(5)
    A, B = _values("all", 0.003, g, outer, M, heads, K).cuda(), _values("all", 0.003, g, outer, N, heads, K).cuda()
    outs = []
    for policy in (2, 1):
        packed.pamk_test_set_packing_policy(policy)
        out = torch.full((outer, heads, M, ld), -7.0, device="cuda")
        ws = torch.empty(packed.pamk_matmul_scratch_bytes(outer * heads, M, N, K, 1) + 256, dtype=torch.uint8, device="cuda")
        _lib.check(packed.pamk_matmul_strided(A.data_ptr(), B.data_ptr(), out.data_ptr(), outer, heads, M, N, K, M * heads * K, K, heads * K, 1,
                                              N * heads * K, K, 1, heads * K, heads * M * ld, M * ld, ld, 1.0, 1, 0.125, 1, ws.data_ptr(),
                                              ws.numel(), torch.cuda.current_stream().cuda_stream), "strided")
        outs.append(out)
    assert_bits_equal(outs[1], outs[0])
    assert bool((outs[1][..., N:] == -7.0).all()) and not bool((outs[1][..., :N] == -7.0).any())


def test_a_large_product_through_the_operators():
    """Above the line where packing pays, through both host paths: the same bits as on the operands as they are."""
    import pam_b200 as pam
    from pam_b200 import _lib, cuda_bindings as cb
    lib = _lib.lib()
    M, N, K = 3200, 3100, 3050
    assert lib.pamk_matmul_scratch_bytes(1, M, N, K, 0) > lib.pamk_matmul_workspace_bytes(1, M, N, lib.pamk_matmul_auto_split(1, M, N, K)) + 255
    g = torch.Generator().manual_seed(8)
    A, B = _values("all", 1e-5, g, M, K).cuda(), _values("below", 1e-3, g, K, N).cuda()
    lib.pamk_test_set_packing_policy(2)
    try:
        want = cb._matmul(_lib.MUL_PAM, A, B, 1.0, 2)
    finally:
        lib.pamk_test_set_packing_policy(0)
    launches = lib.pamk_launch_count()
    assert_bits_equal(cb._matmul(_lib.MUL_PAM, A, B, 1.0, 2), want)
    assert_bits_equal(pam.matmul(A, B), want)
    reduction = lib.pamk_matmul_auto_split(1, M, N, K) > 1
    assert lib.pamk_launch_count() - launches == 2 * (3 + reduction)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = pam.matmul(A, B)
    graph.replay()
    assert_bits_equal(out, want)


@pytest.mark.parametrize("ms", [0, 40, 300])
def test_a_wait_ends_by_the_clock(ms):
    """Barriers that nothing arrives at: the first warp leaves after its limit, the others, whose own is two seconds, with it, and
    one of them is counted."""
    from pam_b200 import _lib
    out = torch.full((10,), 7, dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().pamk_test_run_out(ms, out.data_ptr(), torch.cuda.current_stream().cuda_stream), "run out")
    have = out.tolist()
    assert have[:8] == [0] * 8 and have[9] == 1
    assert ms <= have[8] < ms + 200                         # (a try sleeps for some microseconds)
    assert _lib.lib().pamk_test_run_out(1001, out.data_ptr(), None) == -1
