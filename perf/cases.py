"""The work that a program built on pam_b200 has it do, as cases for timing and comparison.

Each case is a dict of plain values with a "kind":

  linear      one PAM linear layer: forward alone, or forward and backward in either gradient mode
  matmul      one PAM matrix product (batched when batch > 0), forward alone or with both gradients
  ffn         a ReLU feed-forward block: two linear layers around torch.relu, forward and backward
  elementwise PAM multiplication or division with a tensor, a row vector or a number
  layer_norm  PAM LayerNorm
  softmax     PAM softmax over the last dimension, with or without a causal mask
  adam        one PAM Adam step over the parameters of an encoder-decoder transformer
  vit         DeiT-tiny (192 wide, 3 heads, 12 blocks): inference or a training step without the optimizer
  seq2seq     encoder-decoder transformer (512 wide, FFN 1024, 4 heads): the same two

"grad" is "none" (inference), "approx" (approx_bwd=True, the mode of the training runs) or "exact".
All data are fp32, the library's only type.
"""
import math

import torch

import pam_b200 as pam
from pam_b200 import models, optim, steps

DEV = "cuda"

# what special-value inputs hold besides N(0,1): signed zeros, denormals, very large and very small magnitudes
SPECIALS = (0.0, -0.0, 1e-40, -1e-40, 1.4e-45, -1.4e-45, 1e30, -1e30, 1e-30, -1e-30)


def listed():
    return [
        # one sentence of 32 tokens through one projection of a trained model: the smallest call, all latency
        dict(name="linear_infer_32", kind="linear", tokens=32, fin=512, fout=512, bias=True, relu=False, grad="none"),
        # one image through a trained DeiT-tiny: about 150 small launches in a row
        dict(name="vit_infer_1", kind="vit", batch=1, depth=12, train=False),
        # the smallest product of the benchmark's configurations, forward and both gradients
        dict(name="matmul_512", kind="matmul", batch=0, m=512, k=1024, n=512, specials=0.0, grad="approx"),
        # the first MLP layer of DeiT-tiny at batch 64 (64 x 197 tokens), trained with the exact gradients
        dict(name="linear_exact_12608", kind="linear", tokens=12608, fin=192, fout=768, bias=True, relu=False, grad="exact"),
        # the feed-forward block of the 6+6 transformer on its batch of 4096 tokens: half of the activations are zeros
        dict(name="ffn_relu_4096", kind="ffn", tokens=4096, dim=512, hidden=1024, grad="approx"),
        # a large square product of the scaling sweep, with the 1 % special values that the sweep injects
        dict(name="matmul_8192_specials", kind="matmul", batch=0, m=8192, k=8192, n=8192, specials=0.01, grad="none"),
        # the sweep's elementwise product over 2^26 elements, with both gradients
        dict(name="mul_2e26", kind="elementwise", op="mul", rows=65536, cols=1024, other="tensor", grad="approx"),
        # one LayerNorm of DeiT-tiny at batch 64
        dict(name="layer_norm_12608", kind="layer_norm", rows=12608, width=192, grad="approx"),
        # the attention rows of DeiT-tiny at batch 64: 64 x 3 heads x 197 rows of an odd length
        dict(name="softmax_197", kind="softmax", rows=37824, cols=197, causal=False, grad="approx"),
        # the optimizer step of the 6+6 transformer (about 42 million parameters in some 200 tensors)
        dict(name="adam_6_6", kind="adam", vocab=10000, dim=512, ffn=1024, layers=6, decay=0.0),
        # the DeiT-tiny training step at batch 64
        dict(name="vit_step_64", kind="vit", batch=64, depth=12, train=True),
        # the 6+6 transformer's training step on 128 sentence pairs of 32 tokens
        dict(name="seq2seq_step_128", kind="seq2seq", sentences=128, length=32, layers=6, train=True),
    ]


def _spread(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A matrix dimension: a multiple of 64 (as layer widths are), of 4, or any number, the last two often ragged."""
    n = _spread(rng, lo, hi)
    unit = rng.choice((64, 64, 4, 1))
    return max(unit, n // unit * unit)


def draw(rng):
    kind = rng.choice(("linear", "linear", "matmul", "matmul", "ffn", "elementwise", "layer_norm", "softmax", "adam", "vit", "seq2seq"))
    grad = rng.choice(("none", "approx", "approx", "exact"))
    if kind == "linear":
        return dict(kind=kind, tokens=_spread(rng, 1, 16384), fin=_width(rng, 64, 2048), fout=_width(rng, 64, 2048),
                    bias=rng.random() < 0.8, relu=rng.random() < 0.3, grad=grad)
    if kind == "matmul":
        if rng.random() < 0.4:                                  # attention-sized products, one per batch entry and head
            return dict(kind=kind, batch=_spread(rng, 2, 512), m=_spread(rng, 16, 256), k=rng.choice((32, 64, 128, _spread(rng, 16, 256))),
                        n=_spread(rng, 16, 256), specials=0.0, grad=grad)
        m, k, n = (_width(rng, 64, 8192) for _ in range(3))
        # (with gradients three products are formed; the exact ones hold to smaller sizes, as layers do)
        limit = 8192 ** 3 // (1 if grad == "none" else 3 if grad == "approx" else 16)
        while m * k * n > limit:
            m, k, n = max(m // 2, 1), max(k // 2, 1), max(n // 2, 1)
        return dict(kind=kind, batch=0, m=m, k=k, n=n, specials=rng.choice((0.0, 0.01)), grad=grad)
    if kind == "ffn":
        dim = _width(rng, 64, 1024)
        return dict(kind=kind, tokens=_spread(rng, 32, 8192), dim=dim, hidden=dim * rng.choice((2, 4)), grad="approx")
    if kind == "elementwise":
        return dict(kind=kind, op=rng.choice(("mul", "div")), rows=_spread(rng, 1, 65536), cols=_width(rng, 16, 1024),
                    other=rng.choice(("tensor", "row", "number")), grad=grad)
    if kind == "layer_norm":
        return dict(kind=kind, rows=_spread(rng, 1, 65536), width=_width(rng, 64, 1024), grad=grad)
    if kind == "softmax":
        cols = _spread(rng, 8, 1024)
        return dict(kind=kind, rows=cols * max(1, _spread(rng, 16, 1 << 25) // (cols * cols)), cols=cols,
                    causal=rng.random() < 0.3, grad=grad)
    if kind == "adam":
        dim = 64 * rng.randint(2, 8)
        return dict(kind=kind, vocab=_spread(rng, 1000, 10000), dim=dim, ffn=dim * rng.choice((2, 4)) if dim <= 384 else 1024,
                    layers=rng.randint(1, 6), decay=rng.choice((0.0, 0.05)))
    if kind == "vit":
        return dict(kind=kind, batch=_spread(rng, 1, 64), depth=rng.choice((2, 6, 12)), train=rng.random() < 0.6)
    length = rng.randint(8, 48)
    return dict(kind=kind, sentences=_spread(rng, 1, 4096 // length), length=length, layers=rng.choice((1, 3, 6)), train=rng.random() < 0.6)


# ---- inputs --------------------------------------------------------------------------------------------------

def _randn(g, *shape, scale=1.0, grad=False):
    t = torch.randn(*shape, generator=g, device=DEV)
    return (t * scale if scale != 1.0 else t).requires_grad_(grad)


def _with_specials(g, share, *shape, grad=False):
    t = torch.randn(*shape, generator=g, device=DEV)
    count = int(t.numel() * share)
    if count:
        values = torch.tensor(SPECIALS, device=DEV)
        where = torch.randint(0, t.numel(), (count,), generator=g, device=DEV)
        # (one value for each place, so that a place drawn twice holds the same one on every run)
        t.view(-1)[where] = values[where % len(SPECIALS)]
    return t.requires_grad_(grad)


def _linear_module(g, fin, fout, bias, grad):
    with torch.device(DEV):
        layer = pam.Linear(fin, fout, bias=bias, approx_bwd=grad != "exact")
    with torch.no_grad():
        torch.nn.init.trunc_normal_(layer.weight, std=min(0.05, fin ** -0.5), generator=g)
        if bias:
            layer.bias.normal_(std=0.02, generator=g)
    return layer


def _initialise(model, g, std):
    """Weights, biases and gains as they stand early in training."""
    with torch.no_grad():
        for name, p in model.named_parameters():
            if p.dim() > 1:
                scale = p.shape[-1] ** -0.5 if std is None else std
                p.normal_(std=scale, generator=g)
            else:
                p.normal_(std=0.02, generator=g)
                if "norm" in name and name.endswith("weight"):
                    p.add_(1.0)
    return model


_CFG = models.pam_cfgs(approx_bwd=True)


def _adam_shapes(case):
    d, f = case["dim"], case["ffn"]
    attention = [(d, d), (d,)] * 4 + [(d,), (d,)]
    ffn = [(f, d), (f,), (d, f), (d,), (d,), (d,)]
    return [(case["vocab"], d)] * 2 + (attention + ffn) * case["layers"] + (attention * 2 + ffn) * case["layers"]


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind, s = case["kind"], dict(case)
    train = case.get("grad", "none") != "none"
    if kind == "linear":
        x = _randn(g, case["tokens"], case["fin"])
        s["x"] = (torch.relu(x) if case["relu"] else x).requires_grad_(train)
        s["layer"] = _linear_module(g, case["fin"], case["fout"], case["bias"], case["grad"])
        s["gy"] = _randn(g, case["tokens"], case["fout"])
    elif kind == "matmul":
        lead = (case["batch"],) if case["batch"] else ()
        s["a"] = _with_specials(g, case["specials"], *lead, case["m"], case["k"], grad=train)
        s["b"] = _with_specials(g, case["specials"], *lead, case["k"], case["n"], grad=train)
        s["gy"] = _randn(g, *lead, case["m"], case["n"]) if train else None
    elif kind == "ffn":
        s["x"] = _randn(g, case["tokens"], case["dim"], grad=True)
        s["fc1"] = _linear_module(g, case["dim"], case["hidden"], True, case["grad"])
        s["fc2"] = _linear_module(g, case["hidden"], case["dim"], True, case["grad"])
        s["gy"] = _randn(g, case["tokens"], case["dim"])
    elif kind == "elementwise":
        s["a"] = _randn(g, case["rows"], case["cols"], grad=train)
        s["b"] = {"tensor": lambda: _randn(g, case["rows"], case["cols"], grad=train),
                  "row": lambda: _randn(g, case["cols"], grad=train), "number": lambda: 0.125}[case["other"]]()
        s["gy"] = _randn(g, case["rows"], case["cols"])
    elif kind == "layer_norm":
        s["x"] = _randn(g, case["rows"], case["width"], scale=2.0, grad=train)
        s["w"] = (1.0 + _randn(g, case["width"], scale=0.1)).requires_grad_(train)
        s["b"] = _randn(g, case["width"], scale=0.1, grad=train)
        s["gy"] = _randn(g, case["rows"], case["width"])
    elif kind == "softmax":
        x = _randn(g, case["rows"] // case["cols"] if case["causal"] else 1, case["cols"] if case["causal"] else case["rows"], case["cols"])
        if case["causal"]:
            x = x + torch.full((case["cols"], case["cols"]), float("-inf"), device=DEV).triu(1)
        s["x"] = x.requires_grad_(train)
        s["gy"] = _randn(g, *x.shape)
    elif kind == "adam":
        shapes = _adam_shapes(case)
        sizes = [math.prod(shape) for shape in shapes]
        # parameters and moments in one flat buffer each, the tensors views of it, as after loading a checkpoint
        flat = {"p": _randn(g, sum(sizes), scale=0.04), "g": _randn(g, sum(sizes), scale=1e-3),
                "m": _randn(g, sum(sizes), scale=1e-4), "v": _randn(g, sum(sizes), scale=1e-3).square_()}
        views = {name: [t.view(shape) for t, shape in zip(torch.split(buf, sizes), shapes)] for name, buf in flat.items()}
        params = [torch.nn.Parameter(t) for t in views["p"]]
        s["opt"] = optim.Adam(params, lr=5e-4, betas=(0.9, 0.98), weight_decay=case["decay"], opt_functional_cfg="pam")
        for p, grad, m, v in zip(params, views["g"], views["m"], views["v"]):
            p.grad = grad
            s["opt"].state[p] = {"step": 100, "exp_avg": m, "exp_avg_sq": v}
        s["flat"] = flat
    elif kind == "vit":
        cfg = steps.DeitConfig(depth=case["depth"])
        with torch.device(DEV):
            s["model"] = models.VisionTransformer(cfg, linear_cfg=_CFG["linear"], conv_cfg=_CFG["linear"], norm_cfg=_CFG["norm"],
                                                  functional_cfg=_CFG["function"])
        _initialise(s["model"], g, 0.02)
        s["params"] = list(s["model"].parameters())
        s["images"] = _randn(g, case["batch"], cfg.channels, cfg.image, cfg.image)
        s["labels"] = torch.randint(0, cfg.classes, (case["batch"],), generator=g, device=DEV)
    else:
        cfg = steps.TransformerConfig(encoder_layers=case["layers"], decoder_layers=case["layers"])
        with torch.device(DEV):
            s["model"] = models.Transformer(cfg, linear_cfg=_CFG["linear"], norm_cfg=_CFG["norm"], functional_cfg=_CFG["function"],
                                            loss_functional_cfg=_CFG["function"])
        _initialise(s["model"], g, None)
        s["params"] = list(s["model"].parameters())
        tokens = lambda: torch.randint(4, cfg.vocab, (case["sentences"], case["length"]), generator=g, device=DEV)
        s["src"], s["target"] = tokens(), tokens()
        s["prev"] = torch.cat([torch.full((case["sentences"], 1), 2, device=DEV), s["target"][:, :-1]], dim=1)
    return s


# ---- one pass --------------------------------------------------------------------------------------------------

def _with_grads(y, inputs, gy):
    return [y.detach(), *torch.autograd.grad(y, inputs, gy)]


def _all_grads(loss, params):
    """The loss and every gradient, the gradients in one flat tensor as a data-parallel program sums them."""
    return [loss.detach(), torch.cat([t.reshape(-1) for t in torch.autograd.grad(loss, params)])]


def run(s):
    kind, grad = s["kind"], s.get("grad")
    if kind == "linear":
        if grad == "none":
            with torch.no_grad():
                return s["layer"](s["x"])
        return _with_grads(s["layer"](s["x"]), [s["x"], *s["layer"].parameters()], s["gy"])
    if kind == "matmul":
        product = pam.bmm if s["batch"] else pam.matmul
        if grad == "none":
            return product(s["a"], s["b"])
        return _with_grads(product(s["a"], s["b"], approx_bwd=grad == "approx"), [s["a"], s["b"]], s["gy"])
    if kind == "ffn":
        y = s["fc2"](torch.relu(s["fc1"](s["x"])))
        return _with_grads(y, [s["x"], *s["fc1"].parameters(), *s["fc2"].parameters()], s["gy"])
    if kind == "elementwise":
        op = pam.mul if s["op"] == "mul" else pam.div
        if grad == "none":
            return op(s["a"], s["b"])
        inputs = [t for t in (s["a"], s["b"]) if isinstance(t, torch.Tensor)]
        return _with_grads(op(s["a"], s["b"], approx_bwd=grad == "approx"), inputs, s["gy"])
    if kind == "layer_norm":
        y = pam.layer_norm(s["x"], (s["width"],), s["w"], s["b"], 1e-6, approx_bwd=grad == "approx")
        return y if grad == "none" else _with_grads(y, [s["x"], s["w"], s["b"]], s["gy"])
    if kind == "softmax":
        y = pam.softmax(s["x"], dim=-1, approx_bwd=grad == "approx")
        return y if grad == "none" else _with_grads(y, [s["x"]], s["gy"])
    if kind == "adam":
        s["opt"].step()
        return [s["flat"]["p"], s["flat"]["m"], s["flat"]["v"]]
    if kind == "vit":
        if not s["train"]:
            with torch.no_grad():
                return s["model"](s["images"])
        return _all_grads(torch.nn.functional.cross_entropy(s["model"](s["images"]), s["labels"]), s["params"])
    if not s["train"]:
        with torch.no_grad():
            return s["model"](s["src"], s["prev"])
    return _all_grads(s["model"].loss(s["src"], s["prev"], s["target"], fused=True), s["params"])


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def _product(batch, m, k, n, grad):
    """A product counts one integer add and one fp32 add per multiply-accumulate; each gradient forms as many again."""
    a, b, c = batch * m * k, batch * k * n, batch * m * n
    if grad == "none":
        return 4 * (a + b + c), 2 * batch * m * k * n
    return 4 * (2 * a + 2 * b + 2 * c), 6 * batch * m * k * n


def work(case):
    kind, grad = case["kind"], case.get("grad", "none")
    if kind == "linear":
        b, f = _product(1, case["tokens"], case["fin"], case["fout"], grad)
    elif kind == "matmul":
        b, f = _product(max(case["batch"], 1), case["m"], case["k"], case["n"], grad)
    elif kind == "ffn":
        b, f = (u + v for u, v in zip(_product(1, case["tokens"], case["dim"], case["hidden"], grad),
                                      _product(1, case["tokens"], case["hidden"], case["dim"], grad)))
        b += 4 * 4 * case["tokens"] * case["hidden"]                    # the ReLU and its gradient
    elif kind == "elementwise":
        n, second = case["rows"] * case["cols"], case["other"] == "tensor"
        b = 4 * n * (2 + second) + (0 if grad == "none" else 4 * n * (2 + 2 * second))
        f = n * (1 if grad == "none" else 2 + (case["other"] != "number"))
    elif kind == "layer_norm":
        n = case["rows"] * case["width"]
        b, f = (8 * n, 8 * n) if grad == "none" else (20 * n, 24 * n)
    elif kind == "softmax":
        n = case["rows"] * case["cols"]
        b, f = (8 * n, 6 * n) if grad == "none" else (20 * n, 16 * n)
    elif kind == "adam":
        n = sum(math.prod(shape) for shape in _adam_shapes(case))
        b, f = 28 * n, 16 * n
    elif kind == "vit":
        cfg = steps.DeitConfig(depth=case["depth"])
        macs, weights = steps.deit_macs(cfg, case["batch"]), 445_000 * case["depth"] + 186_000
        pixels = case["batch"] * cfg.channels * cfg.image ** 2
        b = 4 * (pixels + weights * (2 if case["train"] else 1))
        f = 2 * macs * (3 if case["train"] else 1)
    else:
        cfg = steps.TransformerConfig(encoder_layers=case["layers"], decoder_layers=case["layers"])
        macs = steps.transformer_macs(cfg, case["sentences"], case["length"])
        weights = 2 * cfg.vocab * cfg.dim + case["layers"] * 5_260_000
        logits = case["sentences"] * case["length"] * cfg.vocab
        b = 4 * (weights * 2 if case["train"] else weights + logits)
        f = 2 * macs * (3 if case["train"] else 1)
    return {"bytes": b, "flops": f}


def tolerance(case):
    kind = case["kind"]
    if kind == "adam" or (kind == "elementwise" and case["other"] != "row"):
        return "exact"                       # no sums: every value is the bit pattern that the definition gives
    if kind == "vit":
        return {"rel": 2e-5}                 # 12 blocks of 32-bit sums, each block carrying on the last one's rounding
    if kind == "seq2seq" and case["train"]:
        # A ReLU input within rounding of zero opens or shuts its unit: the gradients of two orders of summation
        # (K split and unsplit) differ by 2e-4 overall and by 0.03 of the root mean square in single entries.
        return {"rel": 1e-3, "max": 0.1}
    return {"rel": 1e-5}                     # 32-bit sums
