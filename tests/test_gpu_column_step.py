"""The column step without divisions gives the codes of the step with IEEE divisions, bit for bit:
one block of 128 columns (no trailing products) against the same operations in torch fp32."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(w, u, wbits, gs, sym):
    """codes, scales, zeros of one block, every operation rounded to fp32 in the kernel's order"""
    w0 = w.float()
    w = w0.clone()
    out, d = w.shape
    maxq = float(2 ** wbits - 1)
    codes, scales, zeros = torch.empty(out, d, dtype=torch.int32), [], []
    for i in range(d):
        if i % gs == 0:
            lo, hi = w0[:, i:i + gs].amin(1).clamp(max=0), w0[:, i:i + gs].amax(1).clamp(min=0)
            if sym:
                hi = torch.maximum(lo.abs(), hi)
                lo = torch.where(lo < 0, -hi, lo)
            flat = (lo == 0) & (hi == 0)
            lo, hi = torch.where(flat, -torch.ones(()), lo), torch.where(flat, torch.ones(()), hi)
            s = (hi - lo) / maxq
            z = torch.full_like(s, (maxq + 1) / 2) if sym else torch.round(-lo / s)
            scales.append(s)
            zeros.append(z)
        x = w[:, i]
        q = (torch.round(x / s) + z).clamp(0, maxq)
        e = (x - s * (q - z)) / u[i, i]
        codes[:, i] = q.int()
        w[:, i:] = w[:, i:] - e[:, None] * u[i, i:]
    return codes, torch.stack(scales), torch.stack(zeros).int()


@pytest.mark.parametrize("rows", [1, 33, 300, 19000])
@pytest.mark.parametrize("wbits,gs,sym", [(4, 128, False), (3, 32, True), (8, 16, False), (2, 64, False)])
@pytest.mark.parametrize("case", ["random", "ties", "extreme"])
def test_block_of_columns_is_exact(rows, wbits, gs, sym, case):
    from onecompression_b200 import kernels as K

    d = 128
    g = torch.Generator().manual_seed(rows * 10 + wbits)
    w = torch.randn(rows, d, generator=g) * 0.02
    u = torch.triu(torch.randn(d, d, generator=g) * 0.05, 1) + torch.diag(0.5 + torch.rand(d, generator=g))
    if case == "ties":        # half steps of a scale that is a power of two, updates that keep them
        w = torch.randint(0, 2 ** (wbits + 1) - 1, (rows, d), generator=g) * 2.0 ** -10
        w[:, ::gs] = (2 ** wbits - 1) * 2.0 ** -9
        u = torch.diag(torch.ones(d)) + torch.triu(torch.randint(-1, 2, (d, d), generator=g).float(), 1)
        if sym:
            w -= w.mean(1, keepdim=True).mul(2 ** 10).round().div(2 ** 10)
    elif case == "extreme":   # all-zero and subnormal rows, diagonal entries outside the safe range
        w[::3] = 0
        w[1::3] *= 2.0 ** -18
        u[::5, :] = u[::5, :] * 2.0 ** -70
        u[3, 3] = 2.0 ** 70
    w = w.half()
    want = reference(w, u, wbits, gs, sym)
    dev = torch.device("cuda:0")
    iota = torch.arange(d, dtype=torch.int32, device=dev)
    f = K.HessianFactor(u.to(dev), iota, iota, torch.zeros(d, dtype=torch.uint8, device=dev),
                        torch.ones(2, device=dev), False, 0.01, 1.0, 1)
    got = K.gptq_quantize(w.to(dev), f, wbits, gs, sym, pack=False, want_codes=True, want_scales_f32=True)
    assert torch.equal(got["scales_f32"].cpu(), want[1])
    assert torch.equal(got["zeros"].cpu(), want[2])
    assert torch.equal(got["codes"].cpu(), want[0])


@pytest.mark.parametrize("rows", [8, 19000])
def test_group_whose_scale_rounds_to_zero(rows):
    """The zero point is infinite: the first code is the top one, and NaNs follow, for few rows as for many."""
    from onecompression_b200 import kernels as K

    d = 256
    dev = torch.device("cuda:0")
    w = torch.zeros(rows, d)
    w[:, 0], w[:, 1] = 1.25, 15.0                  # scale 1, zero point 0, an error of 1/4 in column 0
    u = torch.eye(d)
    u[0, 128], u[0, 129] = -2.0 ** -147, 2.0 ** -147    # the second group: 2^-149, -2^-149, 0, 0, ...
    iota = torch.arange(d, dtype=torch.int32, device=dev)
    f = K.HessianFactor(u.to(dev), iota, iota, torch.zeros(d, dtype=torch.uint8, device=dev),
                        torch.ones(2, device=dev), False, 0.01, 1.0, 1)
    old = K._lib.load().oc_set_gemm_engine(1)      # the FMA engine keeps subnormal values
    try:
        got = K.gptq_quantize(w.half().to(dev), f, 4, 128, False, pack=False, want_codes=True, want_scales_f32=True)
    finally:
        K._lib.load().oc_set_gemm_engine(old)
    want = torch.zeros(rows, d, dtype=torch.int32)
    want[:, 0], want[:, 1], want[:, 128] = 1, 15, 15
    assert not got["scales_f32"][1].any()
    assert torch.equal(got["codes"].cpu(), want)


@pytest.mark.parametrize("gs,act", [(48, False), (48, True), (80, False), (256, True), (256, False), (-1, False)])
@pytest.mark.parametrize("mse", [False, True])
def test_groups_across_blocks_do_not_depend_on_the_kernel(gs, act, mse):
    """A group that crosses the end of a block, or holds several blocks, has its parameters handed between
    the warps of the window kernel and from block to block.  96 rows take that kernel, 9600 the general one."""
    from onecompression_b200 import kernels as K

    d, out, dev = 640, 9600, torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(gs + 100)
    x = torch.randn(2048, d, generator=g, device=dev).half()
    x[:, ::37] *= 6
    f = K.factor_hessian(K.hessian_from_activations(x)[0], 0.01, act)
    w = (torch.randn(out, d, generator=g, device=dev) * 0.02).half()
    args = dict(wbits=3, groupsize=gs, sym=False, pack=False, want_codes=True, want_scales_f32=True, mse=mse, q_grid=20)
    whole = K.gptq_quantize(w, f, **args)
    for r0 in (0, 4800, 9504):
        part = K.gptq_quantize(w[r0:r0 + 96].contiguous(), f, **args)
        for name in ("codes", "dequantized"):
            assert torch.equal(part[name], whole[name][r0:r0 + 96])
        for name in ("scales_f32", "scales", "zeros"):
            assert torch.equal(part[name], whole[name][:, r0:r0 + 96])
