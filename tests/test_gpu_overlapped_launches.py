"""Kernels that are set up while the one before them still runs (the reduction of a product's ranges, the second halves of column sums and of
LayerNorm's parameter gradients, softmax behind its maximum pass): many operators in a row on changing data, without a
synchronisation and replayed from a captured graph, give what each gives alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operators(x, w, ln, g):
    """Products in ranges, a bias gradient, LayerNorm's gradients, softmax over the results: each reads what the last one wrote."""
    import pam_b200 as pam
    y = pam.matmul(x, w)                                       # in ranges of K
    h = ln(y)
    p = pam.softmax(h * 0.5, dim=-1)
    dx, dw, db, *rest = torch.autograd.grad(p, [x, w, ln.weight, ln.bias], g)
    return [y, h, p, dx, dw, db, *rest]


def _setup(rows, n, k, seed):
    import pam_b200 as pam
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(rows, k, device="cuda", generator=g).requires_grad_()
    w = (torch.randn(k, n, device="cuda", generator=g) * k ** -0.5).requires_grad_()
    with torch.device("cuda"):
        ln = pam.LayerNorm(n, approx_bwd=True)
    return x, w, ln, torch.randn(rows, n, device="cuda", generator=g)


SHAPES = [(512, 512, 1024), (197, 192, 768), (33, 197, 2000), (2048, 64, 640)]


@pytest.mark.parametrize("rows,n,k", SHAPES)
def test_in_a_row(rows, n, k):
    from pam_b200 import _lib
    assert _lib.lib().pamk_matmul_auto_split(1, rows, n, k) > 1
    data = [_setup(rows, n, k, seed) for seed in range(6)]
    alone = []
    for d in data:
        alone.append([t.clone() for t in _operators(*d)])
        torch.cuda.synchronize()
    for _ in range(5):
        for outs, wants in zip([_operators(*d) for d in data], alone):
            for have, want in zip(outs, wants):
                assert torch.equal(have, want)


@pytest.mark.parametrize("rows,n,k", SHAPES[:2])
def test_in_a_captured_graph(rows, n, k):
    x, w, ln, g = _setup(rows, n, k, 1)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _operators(x, w, ln, g)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = _operators(x, w, ln, g)
    for seed in (2, 3):
        other = _setup(rows, n, k, seed)
        with torch.no_grad():
            x.copy_(other[0]), w.copy_(other[1]), g.copy_(other[3])
        graph.replay()
        for have, want in zip(outs, _operators(*other)):
            assert torch.equal(have, want)


@pytest.mark.parametrize("rows,cols", [(12608, 192), (4096, 1024), (70, 33)])
def test_bias_gradients(rows, cols):
    from pam_b200 import cuda_bindings as cb
    xs = [torch.randn(rows, cols, device="cuda") for _ in range(8)]
    alone = []
    for x in xs:
        alone.append(cb._column_sum(x).clone())
        torch.cuda.synchronize()
    for _ in range(5):
        for have, want in zip([cb._column_sum(x) for x in xs], alone):
            assert torch.equal(have, want)
