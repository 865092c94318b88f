"""Performance cases of layer quantization, each a call that a program using this package makes.

The kinds follow the path of one Linear layer: second moments of its activations, the
inverse-Hessian factor, the weight correction, the column loop, and the packed layer that comes
out; a small layer and a mixture's experts go through the whole call.  Sizes are the decoder
shapes of ``onecompression_b200/synthetic.py`` (hidden 4096 / 5120, intermediate 14336), the
2880-wide experts of the tests and the benchmark, and generic ones.
"""

import math

import torch

from onecompression_b200 import GPTQ, kernels
from onecompression_b200.quantizer.gptq._gptq import run_gptq
from onecompression_b200.quantizer.gptq.gptq_layer import GPTQLinear

BLOCK = 128
PERCDAMP = 0.01


def listed():
    return [
        # one small layer through the functional call: launches, synchronisations and host work
        dict(name="layer_small", kind="layer", out=128, d=256, bits=4, gs=128, sym=False, act=False, dtype="fp16"),
        # the Hessian of an attention input, the eight sequences that one update takes
        dict(name="hessian_4096", kind="hessian", d=4096, seqs=8, tokens=2048, dtype="fp16"),
        # one expert's Hessian from the ragged number of tokens that were routed to it
        dict(name="hessian_expert", kind="hessian", d=2880, seqs=1, tokens=1037, dtype="bf16"),
        # Hessian and cross term of the weight correction, as the block driver accumulates them
        dict(name="moments_cross", kind="cross", d=5120, seqs=4, tokens=2048, dtype="bf16"),
        # the factor that the layers of one group share: hidden-sized, and the widest (down_proj)
        dict(name="factor_4096", kind="factor", d=4096, act=False),
        dict(name="factor_14336", kind="factor", d=14336, act=True),
        # weight correction of one attention projection
        dict(name="correct_4096", kind="correct", out=4096, d=4096, dtype="fp16"),
        # the column loop: one projection, the stacked gate / up pair, the widest layer
        dict(name="columns_4096", kind="columns", out=4096, d=4096, bits=3, gs=128, sym=False, act=False, dtype="fp16"),
        dict(name="columns_tall", kind="columns", out=28672, d=4096, bits=4, gs=128, sym=True, act=False, dtype="fp16"),
        dict(name="columns_wide", kind="columns", out=4096, d=14336, bits=4, gs=128, sym=False, act=True, dtype="bf16"),
        # experts of a mixture, each with a Hessian of its own, as one batch
        dict(name="experts", kind="experts", batch=8, out=2880, d=2880, bits=4, gs=32, sym=True, dtype="bf16"),
        # the packed layer at work on a few tokens
        dict(name="linear_decode", kind="linear", out=14336, d=4096, tokens=4, bits=4, gs=128, act=False),
    ]


def _log(rng, lo, hi, step):
    """A multiple of ``step`` between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["layer", "hessian", "cross", "factor", "correct", "columns", "experts", "linear"])
    case = dict(kind=kind)
    if kind in ("layer", "columns", "experts"):
        # (8 bits only where the factor is given: their codes are too fine to survive another rounding of it)
        case.update(bits=rng.choice([2, 3, 4, 4, 8] if kind == "columns" else [2, 3, 4, 4]),
                    gs=rng.choice([32, 64, 128, 128, -1]), sym=rng.random() < 0.5, dtype=rng.choice(["fp16", "bf16"]))
    if kind == "layer":
        case.update(out=_log(rng, 32, 1024, 32), d=_log(rng, 64, 1024, 32), act=rng.random() < 0.5)
    elif kind == "hessian":
        case.update(d=_log(rng, 256, 14336, 8), seqs=rng.choice([1, 2, 4, 8]), tokens=_log(rng, 24, 2048, 1),
                    dtype=rng.choice(["fp16", "bf16"]))
    elif kind == "cross":
        case.update(d=_log(rng, 512, 8192, 8), seqs=rng.choice([1, 2, 4]), tokens=_log(rng, 64, 2048, 1),
                    dtype=rng.choice(["fp16", "bf16"]))
    elif kind == "factor":
        case.update(d=_log(rng, 256, 14336, 4), act=rng.random() < 0.5)
    elif kind == "correct":
        case.update(out=_log(rng, 256, 14336, 8), d=_log(rng, 512, 5120, 8), dtype=rng.choice(["fp16", "bf16"]))
    elif kind == "columns":
        case.update(out=_log(rng, 256, 28672, 32), act=rng.random() < 0.5)
        case.update(d=_log(rng, 512, 14336 if case["out"] <= 4096 else 4096, 32))
    elif kind == "experts":
        case.update(batch=rng.randint(2, 8), out=_log(rng, 512, 2880, 32), d=_log(rng, 512, 2880, 32))
    else:
        case.update(out=_log(rng, 512, 14336, 32), d=_log(rng, 512, 14336, 32), tokens=_log(rng, 1, 4096, 1),
                    bits=rng.choice([2, 3, 4, 4, 8]), gs=rng.choice([32, 64, 128, -1]), act=rng.random() < 0.5)
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(g, rows, d, dtype, outliers=8):
    """N(0, 1) features, a common low-rank part and a few channels twenty times as large."""
    x = torch.randn(rows, d, generator=g, device="cuda")
    rank = 32
    x += 0.5 * torch.randn(rows, rank, generator=g, device="cuda") @ (
        torch.randn(rank, d, generator=g, device="cuda") / math.sqrt(rank))
    x[:, torch.randperm(d, generator=g, device="cuda")[:outliers]] *= 20
    return x.to(dtype)


def _weight(g, out, d, dtype):
    return (0.02 * torch.randn(out, d, generator=g, device="cuda")).to(dtype)


def _hessian(g, d):
    """(2/N) X^T X of 2·d tokens (at least 1024, at most 16384) in fp32."""
    x = _activations(g, max(1024, min(16384, 2 * d)), d, torch.float16).float()
    return torch.mm(x.t(), x).mul_(2.0 / x.shape[0])


def _permutation(h, act):
    d = h.shape[0]
    return torch.argsort(torch.diagonal(h), descending=True, stable=True) if act else torch.arange(d, device=h.device)


def _factor64(h, act):
    """(U, perm) in 64 bits: U upper with U^T U = (P H P^T + damp I)^-1."""
    perm = _permutation(h, act)
    a = h.double()[perm][:, perm]
    diag = torch.diagonal(a)
    diag[diag == 0] = 1.0
    diag += PERCDAMP * diag.mean()
    a = torch.cholesky_inverse(torch.linalg.cholesky(a))
    return torch.linalg.cholesky(a, upper=True), perm


def _ready_factor(h, act):
    """The factor a program keeps for the layers of a group."""
    u, perm = _factor64(h, act)
    d = h.shape[0]
    mean = torch.diagonal(h).mean()
    return kernels.HessianFactor(
        u=u.float().contiguous(), perm=perm.int(), invperm=torch.argsort(perm).int(),
        dead=torch.zeros(d, dtype=torch.uint8, device="cuda"), damp=torch.stack([PERCDAMP * mean, mean]).float(),
        actorder=act, percdamp=PERCDAMP, rel_shift=1.0, attempts=1)


def _layer(weight):
    lin = torch.nn.Linear(weight.shape[1], weight.shape[0], bias=False, device="meta")
    lin.weight = torch.nn.Parameter(weight, requires_grad=False)
    return lin


def _groups(case):
    return 1 if case["gs"] == -1 else (case["d"] + case["gs"] - 1) // case["gs"]


def prepare(case, seed):
    g = _generator(seed)
    kind, d = case["kind"], case["d"]
    dtype = _DTYPES[case.get("dtype", "fp16")]
    if kind == "hessian":
        x = _activations(g, case["seqs"] * case["tokens"], d, dtype).view(case["seqs"], case["tokens"], d)
        lin = torch.nn.Linear(d, 8, bias=False, device="cuda", dtype=dtype)
        return dict(kind=kind, quantizer=GPTQ(), layer=lin, x=x)
    if kind == "cross":
        xf = _activations(g, case["seqs"] * case["tokens"], d, dtype)
        xq = (xf * (1 + 0.05 * torch.randn(xf.shape, generator=g, device="cuda"))).to(dtype)
        shape = (case["seqs"], case["tokens"], d)
        return dict(kind=kind, d=d, xf=xf.view(shape), xq=xq.view(shape))
    if kind == "factor":
        return dict(kind=kind, h=_hessian(g, d), act=case["act"])
    if kind == "layer":
        return dict(kind=kind, h=_hessian(g, d), layer=_layer(_weight(g, case["out"], d, dtype)),
                    args=dict(wbits=case["bits"], groupsize=case["gs"], sym=case["sym"], actorder=case["act"],
                              percdamp=PERCDAMP))
    if kind == "correct":
        w, h = _weight(g, case["out"], d, dtype), _hessian(g, d)
        c = 0.02 * h + torch.randn(d, d, generator=g, device="cuda") * (0.05 * torch.diagonal(h).mean() / math.sqrt(d))
        return dict(kind=kind, w=w, c=c, factor=_ready_factor(h, False))
    if kind == "columns":
        w, h = _weight(g, case["out"], d, dtype), _hessian(g, d)
        return dict(kind=kind, w=w, factor=_ready_factor(h, case["act"]),
                    args=dict(wbits=case["bits"], groupsize=case["gs"], sym=case["sym"]))
    if kind == "experts":
        layers = [_layer(_weight(g, case["out"], d, dtype)) for _ in range(case["batch"])]
        quantizer = GPTQ(wbits=case["bits"], groupsize=case["gs"], sym=case["sym"], percdamp=PERCDAMP,
                         bitpack_on_quantize=False)
        quantizer.module_to_name = {layer: "expert.%d" % i for i, layer in enumerate(layers)}
        return dict(kind=kind, quantizer=quantizer, items=[(layer, _hessian(g, d)) for layer in layers])
    codes, scale, zero, perm = _linear_parts(case, g)
    layer = GPTQLinear(d, case["out"], case["bits"], case["gs"], case["act"], codes, scale, zero, perm=perm)
    return dict(kind=kind, layer=layer, x=_activations(g, case["tokens"], d, torch.float16))


def _linear_parts(case, g):
    out, d, top = case["out"], case["d"], (1 << case["bits"]) - 1
    groups = _groups(case)
    codes = torch.randint(0, top + 1, (out, d), generator=g, device="cuda", dtype=torch.int32)
    scale = ((0.5 + torch.rand(groups, out, generator=g, device="cuda")) * (0.08 / (top + 1))).half()
    zero = torch.randint(1, top + 1, (groups, out), generator=g, device="cuda", dtype=torch.int32)
    perm = torch.randperm(d, generator=g, device="cuda") if case["act"] else None
    return codes, scale, zero, perm


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "hessian":
        return state["quantizer"].calculate_hessian(state["layer"], state["x"])[0]
    if kind == "cross":
        acc = kernels.MomentAccumulator(state["d"], state["xq"].device, cross=True)
        for xq, xf in zip(state["xq"].split(2), state["xf"].split(2)):
            acc.add(xq, xf)
        h, c, _ = acc.finalize()
        return [h, c]
    if kind == "factor":
        f = kernels.factor_hessian(state["h"], PERCDAMP, state["act"])
        return dict(u=f.u, perm=f.perm, invperm=f.invperm, dead=f.dead, damp=f.damp)
    if kind == "layer":
        res = run_gptq(state["h"], state["layer"], **state["args"])
        return {k: v for k, v in res.items() if v is not None}
    if kind == "correct":
        return kernels.qep_adjust(state["w"].clone(), state["c"], state["factor"], 0.5)
    if kind == "columns":
        return kernels.gptq_quantize(state["w"], state["factor"], **state["args"])
    if kind == "experts":
        # (the propagated weight is a function of these three)
        return [{k: one[k] for k in ("codes", "zeros", "scales")}
                for one in state["quantizer"].independent_on_device(state["items"])]
    return state["layer"](state["x"])


def work(case):
    kind, d = case["kind"], case["d"]
    rows = case.get("seqs", 1) * case.get("tokens", 1)
    if kind == "hessian":    # symmetric: half of the products
        return {"bytes": 2.0 * rows * d + 4.0 * d * d, "flops": 1.0 * rows * d * d}
    if kind == "cross":
        return {"bytes": 4.0 * rows * d + 8.0 * d * d, "flops": 3.0 * rows * d * d}
    if kind == "factor":     # Cholesky and triangular inverse
        return {"bytes": 8.0 * d * d, "flops": 2.0 / 3.0 * d ** 3}
    out = case["out"]
    if kind == "linear":
        return {"bytes": out * d * case["bits"] / 8 + _groups(case) * out * (2 + case["bits"] / 8)
                + 2.0 * rows * (out + d), "flops": 2.0 * rows * out * d}
    if kind == "correct":    # one dense and two triangular products
        return {"bytes": 4.0 * out * d + 4.0 * d * d + 2.0 * d * d, "flops": 4.0 * out * d * d}
    # the column loop: weight in, upper triangle of the factor, packed codes, parameters, weight out
    loop = 4.0 * out * d + 2.0 * d * d + out * d * case["bits"] / 8 + _groups(case) * out * (2 + case["bits"] / 8)
    flops = 1.0 * out * d * d
    if kind == "columns":
        return {"bytes": loop, "flops": flops}
    loop += 4.0 * out * d     # plain integer codes
    return {"bytes": case.get("batch", 1) * (loop + 4.0 * d * d), "flops": case.get("batch", 1) * (flops + 2.0 / 3.0 * d ** 3)}


# ---------------------------------------------------------------------------
# what the outputs are held against
# ---------------------------------------------------------------------------


def tolerance(case):
    kind = case["kind"]
    if kind in ("hessian", "cross"):
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "factor":
        return {"rel": 1e-4, "max": 2e-2, "differ": 1e-3}
    if kind == "correct":
        return {"rel": 1e-3 if case["dtype"] == "fp16" else 7e-3, "max": 2e-2}
    if kind == "linear":
        return {"rel": 1e-3, "max": 1e-2}
    # A weight close to the middle between two codes takes either, and what follows in its row moves:
    # up to 0.3 % of the codes differ from those of the same steps in 64 bits, where each rounds the factor itself.
    return {"rel": 0.03, "max": 0.99, "differ": 0.01}


def _parameters64(v, case):
    """(scale, zero) of the rows of v."""
    top = float((1 << case["bits"]) - 1)
    lo, hi = v.amin(1).clamp(max=0), v.amax(1).clamp(min=0)
    if case["sym"]:
        hi = torch.maximum(lo.abs(), hi)
        lo = torch.where(lo < 0, -hi, lo)
    flat = (lo == 0) & (hi == 0)
    lo, hi = torch.where(flat, -1.0, lo), torch.where(flat, 1.0, hi)
    scale = (hi - lo) / top
    zero = torch.full_like(scale, (top + 1) / 2) if case["sym"] else torch.round(-lo / scale)
    return scale, zero


def _columns64(weight, u, perm, case):
    """The column loop in 64 bits: (scales [G, out], W^ [out, d] in original column order)."""
    w = weight.double()[:, perm]
    out, d = w.shape
    top, gs = (1 << case["bits"]) - 1, case["gs"]
    scales, deq = [], torch.empty_like(w)
    scale = zero = None
    if gs == -1:
        scale, zero = _parameters64(weight.double(), case)
        scales.append(scale)
    for i1 in range(0, d, BLOCK):
        i2 = min(d, i1 + BLOCK)
        blk, err = w[:, i1:i2].clone(), torch.zeros(out, i2 - i1, dtype=w.dtype, device=w.device)
        for i in range(i2 - i1):
            if gs != -1 and (i1 + i) % gs == 0:
                scale, zero = _parameters64(w[:, i1 + i:i1 + i + gs], case)
                scales.append(scale)
            x = blk[:, i]
            level = (torch.round(x / scale) + zero).clamp_(0, top).sub_(zero)
            deq[:, i1 + i] = scale.half().double() * level
            e = (x - scale * level) / u[i1 + i, i1 + i]
            blk[:, i:].addr_(e, u[i1 + i, i1 + i:i2], alpha=-1)
            err[:, i] = e
        w[:, i2:].addmm_(err, u[i1:i2, i2:], alpha=-1)
    return torch.stack(scales), deq[:, torch.argsort(perm)]


def exact(case, seed):
    state = prepare(case, seed)
    kind = case["kind"]
    if kind in ("hessian", "cross"):
        d, n = case["d"], case["seqs"] * case["tokens"]
        xq = state["x" if kind == "hessian" else "xq"].reshape(n, d)
        h = torch.zeros(d, d, dtype=torch.float64, device="cuda")
        c = torch.zeros_like(h) if kind == "cross" else None
        for s in range(0, n, 4096):
            part = xq[s:s + 4096].double()
            h.addmm_(part.t(), part, alpha=2.0 / n)
            if c is not None:
                c.addmm_((state["xf"].reshape(n, d)[s:s + 4096].double() - part).t(), part, alpha=2.0 / n)
        return h if c is None else [h, c]
    if kind == "factor":
        u, _ = _factor64(state["h"], case["act"])
        mean = torch.diagonal(state["h"]).double().mean()
        return dict(u=u, perm=None, invperm=None, dead=None, damp=torch.stack([PERCDAMP * mean, mean]))
    if kind == "correct":
        w, u = state["w"].double(), state["factor"].u.double()
        return w + 0.5 * (((w @ state["c"].double()) @ u.t()) @ u)
    if kind == "linear":
        g = _generator(seed)
        codes, scale, zero, perm = _linear_parts(case, g)
        order = perm if perm is not None else torch.arange(case["d"], device="cuda")
        group = torch.empty_like(order)
        group[order] = torch.arange(case["d"], device="cuda") // (case["d"] if case["gs"] == -1 else case["gs"])
        w = (scale.double()[group].t() * (codes.double() - zero.double()[group].t())).half().double()
        return state["x"].double() @ w.t()
    if kind == "columns":
        f = state["factor"]
        scales, deq = _columns64(state["w"], f.u.double(), f.perm.long(), case)
        return dict(qweight=None, qzeros=None, scales=scales, zeros=None, dequantized=deq)
    if kind == "layer":
        u, perm = _factor64(state["h"], case["act"])
        scales, _ = _columns64(state["layer"].weight.data, u, perm, case)
        res = dict(qweight=None, scales=scales.t() if case["gs"] == -1 else scales, qzeros=None)
        return dict(res, perm=None) if case["act"] else res
    res = []
    for layer, h in state["items"]:
        u, perm = _factor64(h, False)
        res.append(dict(codes=None, zeros=None, scales=_columns64(layer.weight.data, u, perm, case)[0]))
    return res
