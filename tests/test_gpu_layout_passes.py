"""The passes that bring matrices into and out of the column loop, the factor and the correction: odd
sizes, strided rows and act-order, each against an equivalent call whose passes take another branch (the
column loop between them is the same on both sides)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def spd(n, seed=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(2 * n + 16, n, generator=g, dtype=torch.float64)
    h = (x.t() @ x / len(x) * (0.5 + torch.rand(n, generator=g, dtype=torch.float64))).float()
    return ((h + h.t()) / 2).to(DEV)


@pytest.mark.parametrize("n", [1, 3, 4, 127, 130, 256, 388, 1031, 1160])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_factor_layouts(n, pad):
    """Act-order equals the plain factor of the permuted matrix, whatever the row stride."""
    from onecompression_b200 import kernels as K

    h = spd(n, n)
    if n > 3:
        h[2, :] = h[:, 2] = 0
    wide = torch.full((n, n + pad), float("nan"), device=DEV)
    wide[:, :n] = h
    f = K.factor_hessian(wide[:, :n], 0.01, True)
    p = f.perm.long()
    fixed = h + torch.diag((torch.diagonal(h) == 0).float())
    assert torch.equal(p, torch.argsort(torch.diagonal(fixed), descending=True, stable=True))
    plain = K.factor_hessian(h[p][:, p].contiguous(), 0.01, False)
    assert torch.equal(f.u, plain.u) and torch.equal(f.u, torch.triu(f.u))
    a = fixed.double()[p][:, p] + 0.01 * torch.diagonal(fixed).double().mean() * torch.eye(n, device=DEV)
    want = torch.linalg.cholesky(torch.linalg.inv(a), upper=True)
    assert ((f.u.double() - want).norm() / want.norm()).item() < 2e-5
    if n <= 388:
        two = K.factor_hessians_batched(torch.stack([h, h]).contiguous(), 0.01, True)
        assert torch.equal(two["u"][0], f.u) and torch.equal(two["u"][1], f.u)


@pytest.mark.parametrize("out,d,bits,gs", [(1, 8, 5, -1), (63, 130, 5, 32), (65, 257, 3, -1), (64, 160, 3, 32),
                                           (96, 1056, 2, 48), (130, 264, 8, 128), (100, 516, 7, 64), (72, 392, 4, 128)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("pad", [0, 1, 8])
def test_column_loop_layouts(out, d, bits, gs, dtype, pad):
    from onecompression_b200 import kernels as K

    g = torch.Generator().manual_seed(out + d)
    wide = torch.randn(out, d + pad, generator=g).mul(0.02).to(dtype).to(DEV)
    w = wide[:, :d]
    f = K.factor_hessian(spd(d, 1), 0.01, True)
    f.dead[1::7] = 1
    p = f.perm.long()
    args = dict(wbits=bits, groupsize=gs, sym=False, pack=False, want_codes=True, want_scales_f32=True)
    got = K.gptq_quantize(w, f, **args)
    # the permuted problem without act-order
    iota = torch.arange(d, dtype=torch.int32, device=DEV)
    plain = K.HessianFactor(f.u, iota, iota, f.dead[p].contiguous(), f.damp, False, 0.01, 1.0, 1)
    ref = K.gptq_quantize(w[:, p].contiguous(), plain, **args)
    assert torch.equal(got["codes"][:, p], ref["codes"])
    assert torch.equal(got["dequantized"][:, p], ref["dequantized"])
    assert torch.equal(got["scales_f32"], ref["scales_f32"]) and torch.equal(got["zeros"], ref["zeros"])
    group = torch.arange(d, device=DEV) // (d if gs == -1 else gs)
    s, z = ref["scales"][group].t().float(), ref["zeros"][group].t().float()
    assert torch.equal(ref["dequantized"], (s * (ref["codes"].float() - z)).half().to(dtype))
    f_pack = 32 if bits == 3 else 32 // bits
    if bits in K.PACKABLE_WBITS and d % f_pack == 0 and out % f_pack == 0:
        packed = K.gptq_quantize(w, f, bits, gs, False)
        assert torch.equal(packed["qweight"], K.pack_qweight(got["codes"], bits))
        assert torch.equal(packed["dequantized"], got["dequantized"])


@pytest.mark.parametrize("out,d", [(3, 6), (33, 130), (64, 256), (40, 516)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("pad", [0, 1, 4])
@pytest.mark.parametrize("act", [False, True])
def test_correction_layouts(out, d, dtype, pad, act):
    from onecompression_b200 import kernels as K

    g = torch.Generator().manual_seed(out + d)
    wide = torch.randn(out, d + pad, generator=g).mul(0.02).to(dtype).to(DEV)
    h = spd(d, 2)
    h[5, :] = h[:, 5] = 0
    c = (0.05 * torch.randn(d, d, generator=g)).to(DEV)
    f = K.factor_hessian(h, 0.01, act)
    p = f.perm.long()
    wz = wide[:, :d].double()
    wz[:, 5] = 0
    u = torch.zeros(d, d, dtype=torch.float64, device=DEV)
    u[:, p] = f.u.double()                       # U P: (H + damp I)^-1 = (U P)^T (U P)
    want = wz + 0.5 * ((wz @ c.double()) @ u.t()) @ u
    before = wide.clone()
    K.qep_adjust(wide[:, :d], c, f, 0.5)
    got = wide[:, :d].double()
    # one rounding to 16 bits of a sum that the products give to about 1e-5
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert ((got - want).abs() <= eps * want.abs() + 1e-5 * want.abs().max()).all()
    assert torch.equal(wide[:, d:], before[:, d:])
