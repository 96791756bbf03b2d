"""One fused Adam step on gradients and moments of every magnitude, against the oracle, bit for bit: elements of ordinary
magnitude leave out the range rules, all others (zeros, denormals, tiny and huge values) keep them.
"""
import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


def _any_magnitude(g, n, lo, hi):
    """Sign and mantissa at random, the exponent field between lo and hi (0 gives denormals), every 17th a zero."""
    bits = torch.randint(0, 1 << 23, (n,), generator=g) + (torch.randint(lo, hi + 1, (n,), generator=g) << 23)
    t = bits.to(torch.int32).view(torch.float32) * torch.where(torch.rand(n, generator=g) < 0.5, -1.0, 1.0)
    t[::17] = 0.0
    return t


@pytest.mark.parametrize("lo,hi", [(0, 40), (60, 72), (90, 130), (182, 192), (20, 230)])
@pytest.mark.parametrize("lr,decay,betas", [(5e-4, 0.0, (0.9, 0.98)), (5e-4, 0.05, (0.9, 0.999)), (1e-9, 0.0, (0.9, 0.98))])
def test_adam_step_at_every_magnitude(lo, hi, lr, decay, betas, oracle):
    from pam_b200 import optim
    g = torch.Generator().manual_seed(lo + hi)
    n = 4099
    p, grad, m, v = _any_magnitude(g, n, 100, 128), _any_magnitude(g, n, lo, hi), _any_magnitude(g, n, lo, hi), _any_magnitude(g, n, lo, hi).abs()
    param = torch.nn.Parameter(p.cuda())
    param.grad = grad.cuda()
    opt = optim.Adam([param], lr=lr, betas=betas, eps=1e-8, weight_decay=decay, opt_functional_cfg="pam")
    opt.state[param] = {"step": 9, "exp_avg": m.cuda(), "exp_avg_sq": v.cuda()}
    opt.step()
    want = oracle.adam_step(p.clone(), grad, m.clone(), v.clone(), step=10, lr=lr, betas=betas, eps=1e-8, weight_decay=decay)
    for got, w, what in zip((param.detach(), opt.state[param]["exp_avg"], opt.state[param]["exp_avg_sq"]), want, "pmv"):
        assert_bits_equal(got, w, what)


@pytest.mark.parametrize("n", [1, 3, 4, 127, 128, 129, 1024, 4099])
@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("zeros", ["none", "one", "rows", "tenth", "all"])
def test_adam_step_where_gradients_are_zero(n, aligned, zeros, oracle):
    """A warp (128 elements) takes the rule without range rules or the full one as a whole: gradients without zeros, with one, with
    blocks of zeros (and moments that were never touched), zeros everywhere between; edges of a warp and of a block."""
    from pam_b200 import optim
    g = torch.Generator().manual_seed(n)
    p, grad, m, v = (torch.randn(n, generator=g) * s for s in (0.04, 1e-3, 1e-4, 1e-3))
    v = v.square()
    zero = {"none": torch.zeros(n), "one": torch.arange(n) == n // 2, "rows": torch.arange(n) // 512 % 2,
            "tenth": torch.rand(n, generator=g) < 0.1, "all": torch.ones(n)}[zeros].bool()
    grad[zero] = 0.0
    if zeros == "rows":
        m[zero], v[zero] = 0.0, 0.0
    first = 0 if aligned else 1
    own = lambda t: torch.cat([torch.zeros(first), t]).cuda()[first:]          # (a float past a 16-byte boundary)
    param = torch.nn.Parameter(own(p))
    param.grad = own(grad)
    opt = optim.Adam([param], lr=5e-4, betas=(0.9, 0.98), eps=1e-8, weight_decay=0.05, opt_functional_cfg="pam")
    opt.state[param] = {"step": 9, "exp_avg": own(m), "exp_avg_sq": own(v)}
    opt.step()
    want = oracle.adam_step(p.clone(), grad, m.clone(), v.clone(), step=10, lr=5e-4, betas=(0.9, 0.98), eps=1e-8, weight_decay=0.05)
    for got, w, what in zip((param.detach(), opt.state[param]["exp_avg"], opt.state[param]["exp_avg_sq"]), want, "pmv"):
        assert_bits_equal(got, w, what)
