"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one or two block calls through the package's public entry points: the single-direction
module (``forward``, and ``block`` with a dropout scale), the functional update with packed
projections and a pair mask, and the bidirectional module.  The listed cases span the token counts
that structure models meet, from a short peptide to a large complex, the channel widths of the pair
stack (128), the template stack (64) and the wide configuration (256), both directions, both
activation types and every kind of mask.
"""

from __future__ import annotations

import math

import torch

from miniworld_engine_b200 import (BidirectionalTriangleMultiplicationB200, TriangleMultiplicationB200,
                                   triangle_multiplicative_update_b200)

_DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def _case(form, n, *, b=1, c=128, h=None, dtype="bf16", outgoing=True, mask="ones", name=None):
    case = {} if name is None else {"name": name}
    case.update(form=form, b=b, n=n, c=c, h=c if h is None else h, dtype=dtype, outgoing=outgoing, mask=mask)
    return case


def listed():
    return [
        # full-precision check of a short chain (the smallest configuration of the benchmark set)
        _case("block", 32, dtype="fp32", name="short_chain_fp32"),
        # a peptide or a small domain during inference: launches and host time are all there is
        _case("module", 64, mask="tail", name="peptide"),
        # training forward of a 256-token crop: row-broadcast dropout scale and residual
        _case("dropout", 256, b=2, mask="tail", name="crop_dropout"),
        # the usual 384-token crop
        _case("module", 384, name="crop_384"),
        # functional form as foreign model code calls it: packed projections, pair mask, odd token count
        _case("functional", 449, outgoing=False, mask="pair", name="functional_odd"),
        # a padded batch element of a medium complex
        _case("block", 768, outgoing=False, mask="tail", name="complex_768_padded"),
        # template pair stack: narrow channels, batched
        _case("module", 512, b=2, c=64, name="template_c64"),
        # wide pair representation, batched
        _case("module", 512, b=2, c=256, name="wide_c256"),
        # bidirectional block of a 384-token crop
        _case("bidirectional", 384, mask="tail", name="bidirectional_384"),
        # bidirectional block whose two directions share the pair width between them (d_hidden = 64)
        _case("bidirectional", 320, h=64, mask="random", name="bidirectional_h64"),
        # full-precision run on an ordinary domain
        _case("module", 256, dtype="fp32", outgoing=False, mask="tail", name="domain_fp32"),
        # outgoing then incoming block on a large complex with scattered unresolved tokens
        _case("chain", 2048, mask="random", name="chain_2048"),
    ]


def _spread(rng, lo, hi):
    """A token count between lo and hi, even over the logarithm; half of them odd or ragged."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5:
        n = n // 8 * 8
    return max(lo, min(hi, n))


def draw(rng):
    form = rng.choice(["module", "module", "block", "dropout", "functional", "width", "bidirectional", "fp32", "chain"])
    outgoing = rng.random() < 0.5
    mask = rng.choice(["none", "ones", "tail", "random"])
    if form == "functional":
        h = rng.choice([128, 128, 64])
        return _case("functional", _spread(rng, 32, 1024 if h == 128 else 448), h=h, outgoing=outgoing,
                     mask=rng.choice(["none", "tail", "pair", "pair"]))
    if form == "bidirectional":
        h = rng.choice([128, 64])
        return _case("bidirectional", _spread(rng, 32, 1024 if h == 128 else 448), h=h, mask=mask)
    if form == "width":
        c = rng.choice([64, 256])
        n = _spread(rng, 32, 1024 if c == 64 else 640)
        return _case(rng.choice(["module", "block", "dropout"]), n, b=rng.choice([1, 2]) if n <= 512 else 1, c=c,
                     outgoing=outgoing, mask=mask)
    if form == "fp32":
        return _case(rng.choice(["module", "block"]), _spread(rng, 16, 256), c=rng.choice([64, 128]), dtype="fp32",
                     outgoing=outgoing, mask=mask)
    n = _spread(rng, 32, 2048)
    return _case(form, n, b=rng.choice([1, 2, 3]) if n <= 512 else 1, outgoing=outgoing, mask=mask)


def _mask(kind, b, n, gen):
    if kind == "none":
        return None
    if kind == "pair":
        return torch.rand(b, n, n, generator=gen, device="cuda") > 0.1
    m = torch.ones(b, n, dtype=torch.bool, device="cuda")
    if kind == "tail":
        m[:, n - n // 10:] = False
    elif kind == "random":
        m = torch.rand(b, n, generator=gen, device="cuda") > 0.05
    return m


def _fill(module, dtype, gen):
    """Parameters of a trained block: Linear weights of the fan-in's scale, affine LayerNorms."""
    module = module.to(device="cuda", dtype=dtype).eval().requires_grad_(False)
    for name, p in module.named_parameters():
        v = torch.randn(p.shape, generator=gen, device="cuda")
        if p.dim() == 2:
            v *= p.shape[1] ** -0.5
        elif name.endswith("weight"):
            v = 1.0 + 0.1 * v
        else:
            v *= 0.1
        p.copy_(v)
    return module


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    b, n, c, h, dtype = case["b"], case["n"], case["c"], case["h"], _DTYPES[case["dtype"]]
    state = {"form": case["form"], "mask": _mask(case["mask"], b, n, gen)}
    if case["form"] == "bidirectional":
        state["blocks"] = [_fill(BidirectionalTriangleMultiplicationB200(c, h), dtype, gen)]
    elif case["form"] == "chain":
        state["blocks"] = [_fill(TriangleMultiplicationB200(c, outgoing=o), dtype, gen) for o in (True, False)]
    elif case["form"] == "functional":
        shapes = ((2 * h, c), (2 * h, c), (c, h), (c, c))
        p_in, g_in, p_out, g_out = ((torch.randn(s, generator=gen, device="cuda") * s[1] ** -0.5).to(dtype) for s in shapes)
        n_in, n_out = ((1.0 + 0.1 * torch.randn(d, generator=gen, device="cuda"),
                        0.1 * torch.randn(d, generator=gen, device="cuda")) for d in (c, h))
        state["direction"] = "outgoing" if case["outgoing"] else "incoming"
        state["weights"] = (*n_in, p_in, g_in, *n_out, p_out, g_out)
    else:
        state["blocks"] = [_fill(TriangleMultiplicationB200(c, outgoing=case["outgoing"]), dtype, gen)]
    state["pair"] = torch.randn(b, n, n, c, generator=gen, device="cuda").to(dtype)
    if case["form"] == "dropout":
        state["scale"] = (torch.rand(b, 1, n, c, generator=gen, device="cuda") > 0.25).to(dtype) / 0.75
    return state


@torch.no_grad()
def run(state):
    form, pair, mask = state["form"], state["pair"], state["mask"]
    if form == "functional":
        return triangle_multiplicative_update_b200(pair, state["direction"], mask, *state["weights"])
    if form == "block":         # the bare update, the caller adds it where it wants it
        return state["blocks"][0].block(pair, mask)
    if form == "dropout":       # module.forward in training mode, with the scale drawn beforehand
        return state["blocks"][0].block(pair, mask, residual=pair, drop_scale=state["scale"])
    for block in state["blocks"]:
        pair = block(pair, mask)
    return pair


def work(case):
    """Each block reads its pair tensor and parameters once and writes its result once; four input
    projections, the output projection, the gate and the contraction are its operations."""
    b, n, c, h = case["b"], case["n"], case["c"], case["h"]
    blocks = 2 if case["form"] == "chain" else 1
    width = 2 * h if case["form"] == "bidirectional" else h
    size = 2 if case["dtype"] == "bf16" else 4
    pos = b * n * n
    weights = (5 * width * c + c * c) * size + 8 * (c + width)
    mask = {"none": 0, "pair": pos}.get(case["mask"], b * n)
    scale = b * n * c * size if case["form"] == "dropout" else 0
    return {"bytes": blocks * (2 * pos * c * size + weights + mask) + scale,
            "flops": blocks * (2 * pos * n * width + 2 * pos * (5 * width * c + c * c))}


def tolerance(case):
    """Four times what the outputs show against the same block in 64 bits (fp32: up to 4.1e-7, single
    values 2.5e-6; bf16: 2.7e-3 with the residual, 4.5e-3 without, single values 4.5e-2), and for bf16
    no more than the 1e-2 that the type is held to."""
    if case["dtype"] == "fp32":
        return {"rel": 1.6e-6, "max": 1e-5}
    return {"rel": 1e-2, "max": 0.18}
