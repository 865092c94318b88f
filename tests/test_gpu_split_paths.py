"""The callers of the split products where their shapes can go wrong: partial blocks and panels, one or two blocks,
16-bit types, act-order, rows and diagonals of very different size."""

import pytest
import torch

from onecompression_b200 import kernels as K

pytestmark = pytest.mark.gpu


def gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def moment(n, seed, tokens=4):
    x = torch.randn(tokens * n, n, generator=gen(seed), device="cuda")
    return x.t() @ x / (tokens * n)


def factor64(h, percdamp, perm):
    a = h.double()[perm][:, perm]
    diag = torch.diagonal(a)
    diag += percdamp * diag.mean()
    return torch.linalg.cholesky(torch.cholesky_inverse(torch.linalg.cholesky(a)), upper=True)


def as_factor(u, h, perm=None):
    n = u.shape[0]
    iota = torch.arange(n, device="cuda")
    p = iota if perm is None else perm
    mean = torch.diagonal(h).mean()
    return K.HessianFactor(u.float().contiguous(), p.int(), torch.argsort(p).int(),
                           torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.stack([0.01 * mean, mean]).float(),
                           perm is not None, 0.01, 1.0, 1)


@pytest.mark.parametrize("act", [False, True])
@pytest.mark.parametrize("n", [128, 129, 255, 256, 257, 384, 513, 777, 1027])
def test_factor(n, act):
    """Bound: n * 2^-24 * cond; the moments of 4 n tokens have a condition of 9."""
    h = moment(n, n)
    f = K.factor_hessian(h, 0.01, act)
    u = factor64(h, 0.01, f.perm.long())
    assert (f.u.double() - u).norm() <= n * 2.0**-24 * 9 * u.norm()
    assert torch.equal(f.u, f.u.triu())
    hs = torch.stack([h, moment(n, n + 5000), h])
    out = K.factor_hessians_batched(hs, 0.01, act)
    assert torch.equal(out["u"][0], f.u) and torch.equal(out["u"][2], f.u) and not out["status"].any()


@pytest.mark.parametrize("n", [300, 640])
def test_factor_of_a_badly_scaled_matrix(n):
    """H = D S D, D over 2^-20 .. 2^20: U D is the factor of S, to the accuracy of S alone."""
    s = moment(n, 1)
    d = torch.exp2(torch.randint(-20, 21, (n,), generator=gen(2), device="cuda").float())
    f = K.factor_hessian(s * d[:, None] * d[None, :], 0.0, False)
    u = factor64(s, 0.0, torch.arange(n, device="cuda"))
    assert (f.u.double() * d.double() - u).norm() <= n * 2.0**-24 * 9 * u.norm()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("act", [False, True])
@pytest.mark.parametrize("out,d", [(1, 128), (5, 129), (40, 96), (128, 256), (130, 390), (300, 257)])
def test_correction(out, d, act, dtype):
    """Within one unit of the weight's type of the float64 result (the rounding to it, where fp32 sums meet a tie),
    and a row does not depend on the others."""
    h = moment(d, 3)
    perm = torch.argsort(torch.diagonal(h), descending=True, stable=True) if act else None
    u = factor64(h, 0.01, perm if act else torch.arange(d, device="cuda"))
    f = as_factor(u, h, perm)
    f.dead[d // 3] = 1
    w = torch.randn(out, d, generator=gen(4), device="cuda") * 0.02
    w[0] *= 2.0**-6
    w = w.to(dtype)
    c = 0.02 * h + 0.01 * torch.randn(d, d, generator=gen(5), device="cuda") / d**0.5
    got = K.qep_adjust(w.clone(), c, f, 0.5)
    w64 = w.double()
    w64[:, d // 3] = 0
    p = f.perm.long()
    u64 = f.u.double()
    delta = torch.empty_like(w64)
    delta[:, p] = ((w64 @ c.double())[:, p] @ u64.t()) @ u64
    want = w64 + 0.5 * delta
    # (fp16 values below 2^-14 are 2^-24 apart)
    ulp = want.abs() * 2.0**-10 + 2.0**-24 if dtype == torch.float16 else want.abs() * 2.0**-7
    ulp = ulp + w64.norm(dim=1, keepdim=True) * 2.0**-24
    assert ((got.double() - want).abs() <= ulp).all()
    for r in {0, out // 2, out - 1}:
        assert torch.equal(K.qep_adjust(w[r:r + 1].clone(), c, f, 0.5)[0], got[r])


@pytest.mark.parametrize("act", [False, True])
@pytest.mark.parametrize("out,d,gs", [(1, 256, 128), (40, 160, 32), (33, 640, 128), (260, 1184, -1), (9600, 288, 32),
                                      (2000, 544, 96)])
def test_column_loop(out, d, gs, act):
    """Against the FMA engine on the same factor: sums in another order move a code where a weight lies next to the
    middle between two, and what follows in its row (one row in fifty here at most)."""
    h = moment(d, 6)
    perm = torch.argsort(torch.diagonal(h), descending=True, stable=True) if act else None
    f = as_factor(factor64(h, 0.01, perm if act else torch.arange(d, device="cuda")), h, perm)
    w = (torch.randn(out, d, generator=gen(7), device="cuda") * 0.02)
    w[out // 2] *= 2.0**-10
    w = w.half()
    new = K.gptq_quantize(w, f, 4, gs, False, pack=False, want_codes=True)
    old_mode = K.set_gemm_engine(1)
    try:
        old = K.gptq_quantize(w, f, 4, gs, False, pack=False, want_codes=True)
    finally:
        K.set_gemm_engine(old_mode)
    moved = (new["codes"] != old["codes"]).any(dim=1)
    assert moved.sum() <= 1 + out // 50
    assert torch.equal(new["dequantized"][~moved], old["dequantized"][~moved])
    r = out // 2
    alone = K.gptq_quantize(w[r:r + 1].contiguous(), f, 4, gs, False, pack=False, want_codes=True)
    assert torch.equal(alone["codes"][0], new["codes"][r])
    assert K.gemm_tc_status() == 0


@pytest.mark.parametrize("n", [257, 640, 1027, 1160])
def test_tile_shapes_give_the_same_bits(n):
    """Wide tiles write a result that goes on as an operand as planes themselves, narrow ones leave that to a pass of its
    own: the same values, whatever the workspace held."""
    h = moment(n, 11)
    f = as_factor(factor64(h, 0.01, torch.arange(n, device="cuda")), h)
    w = torch.randn(333, n, generator=gen(12), device="cuda") * 0.02
    c = 0.02 * h + 0.01 * torch.randn(n, n, generator=gen(13), device="cuda") / n**0.5
    got = {}
    for shape in (1, 2):
        old = K.set_gemm_tile_shape(shape)
        try:
            K._workspace(1 << 26, w.device).fill_(0xff)
            got[shape] = [K.factor_hessian(h, 0.01, False).u, K.factor_hessians_batched(torch.stack([h, h * 3]), 0.01, True)["u"]]
            got[shape] += [K.qep_adjust(w.to(t), c, f, 0.5) for t in (torch.float16, torch.bfloat16)]
        finally:
            K.set_gemm_tile_shape(old)
    for a, b in zip(got[1], got[2]):
        assert torch.equal(a, b) and a.isfinite().all()
    assert K.gemm_tc_status() == 0


def test_an_expired_wait_is_not_retried(monkeypatch):
    """A negative status is a product whose pipeline gave up, not a bad pivot: more damping is no help.  (The status is
    planted behind the call; no kernel waits here.)"""
    planted, calls = [], []
    empty, call = torch.empty, K.call

    def remembers(*args, **kw):
        t = empty(*args, **kw)
        if t.dtype == torch.int32 and t.numel() == 1:
            planted.append(t)
        return t

    def plants(name, *args):
        calls.append(name)
        rc = call(name, *args)
        planted[-1].fill_(-204)
        return rc

    monkeypatch.setattr(K.torch, "empty", remembers)
    monkeypatch.setattr(K, "call", plants)
    with pytest.raises(RuntimeError, match="bounded pipeline wait expired .code 204."):
        K.factor_hessian(moment(256, 1), 0.01, False)
    assert calls == ["oc_hinv_factor"]


def test_under_capture():
    """The chains of dependent launches as a graph, behind a join of two streams and a copy: the bits of the plain calls."""
    n, out = 640, 200
    x = torch.randn(300, n, generator=gen(21), device="cuda").half()
    w = (torch.randn(out, n, generator=gen(22), device="cuda") * 0.02).half()
    c = torch.randn(n, n, generator=gen(23), device="cuda") / n
    host = torch.randn(n, n, generator=torch.Generator().manual_seed(24)).pin_memory()
    noise = torch.empty(n, n, device="cuda")
    side, other = torch.cuda.Stream(), torch.cuda.Stream()

    def body():
        here = torch.cuda.current_stream()
        acc = K.MomentAccumulator(n, "cuda")
        acc.add(x)
        h = acc.finalize(check=False)[0]
        other.wait_stream(here)
        with torch.cuda.stream(other):
            noise.copy_(host, non_blocking=True)
            e = noise * 1e-3
        here.wait_stream(other)
        h = h + torch.diag(e.diagonal().abs())
        p = K.factor_hessian_launch(h, 0.01, True)
        f = K.HessianFactor(p["u"], p["perm"], p["invperm"], p["dead"], p["damp"], True, 0.01, 1.0, 1)
        v = K.qep_adjust(w.clone(), c, f, 0.5)
        q = K.gptq_quantize(v, f, 4, 128, False, want_codes=True)
        return [h, f.u, f.perm, v, p["status"]] + [q[k] for k in sorted(q)]

    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = [t.clone() for t in body()]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = body()
        for _ in range(3):
            for t in got:
                t.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert K.gemm_tc_status() == 0
