"""The packed layer: decoding kernel and the product that decodes on the fly."""

import pytest
import torch
from torch.autograd import forward_ad

pytestmark = pytest.mark.gpu


def layer(out, d, bits, gs, act, bias, seed=0):
    from onecompression_b200.quantizer.gptq.gptq_layer import GPTQLinear

    g = torch.Generator().manual_seed(seed)
    groups = 1 if gs == -1 else (d + gs - 1) // gs
    codes = torch.randint(0, 2 ** bits, (out, d), generator=g, dtype=torch.int32)
    scale = (0.5 + torch.rand(groups, out, generator=g)).half() * 0.01
    zero = torch.randint(1, 2 ** bits, (groups, out), generator=g, dtype=torch.int32)
    perm = torch.randperm(d, generator=g) if act else None
    b = torch.randn(out, generator=g).half() if bias else None
    m = GPTQLinear(d, out, bits, gs, act, codes, scale, zero, perm=perm, bias=b)
    order = perm if act else torch.arange(d)
    grp = torch.empty(d, dtype=torch.long)
    grp[order] = torch.arange(d) // (d if gs == -1 else gs)
    w = (scale.float()[grp].t() * (codes.float() - zero.float()[grp].t())).half()
    return m, w


# out: less than a tile of rows, a tile and a rest; d: one unit, less than a share per warp, a rest of 32
@pytest.mark.parametrize("bits,out,d", [(4, 8, 8), (4, 72, 1048), (4, 136, 4096), (2, 48, 2064), (2, 16, 16),
                                        (3, 32, 32), (3, 96, 1056), (8, 4, 8), (8, 100, 520), (8, 68, 1028)])
@pytest.mark.parametrize("gs,act", [(-1, False), (32, False), (128, True), (24, False), (8, True)])
def test_packed_linear(bits, out, d, gs, act):
    from onecompression_b200 import kernels as K

    for bias in (False, True):
        m, w = layer(out, d, bits, gs, act, bias)
        assert torch.equal(m.dequantized_weight().cpu(), w)
        for tokens in (1, 7, 8, 9, 16, 17):
            x = torch.randn(tokens, d, generator=torch.Generator().manual_seed(tokens)).half()
            want = x.double() @ w.double().t() + (m.bias.double().cpu() if bias else 0)
            taken = m._decoded_in_product(x.cuda()) is not None
            assert taken == (tokens <= K.PACKED_LINEAR_TOKENS and d % 8 == 0)
            got = m(x.cuda()).cpu().double()
            # fp32 sums of d products (d * 2^-24 of the sum of magnitudes) and one rounding to fp16
            bound = d * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t()) + 2.0 ** -11 * want.abs() + 2.0 ** -25
            assert ((got - want).abs() <= bound).all()


def test_packed_linear_keeps_the_general_path():
    """Gradients, function transforms, autocast and unaligned or strided inputs go the way they went."""
    m, w = layer(64, 256, 4, 64, False, False)
    x = torch.randn(4, 256, device="cuda").half()
    assert m._decoded_in_product(x) is not None
    y = m(x)
    xg = x.clone().requires_grad_()
    m(xg).sum().backward()
    assert torch.allclose(xg.grad.float(), w.cuda().float().sum(0).expand(4, -1), rtol=1e-2, atol=1e-2)
    assert torch.allclose(torch.func.vmap(m)(x.unsqueeze(1)).squeeze(1), y, rtol=1e-2, atol=1e-2)
    with forward_ad.dual_level():
        tangent = forward_ad.unpack_dual(m(forward_ad.make_dual(x, x))).tangent
    assert torch.allclose(tangent, y, rtol=1e-2, atol=1e-2)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert m(x).dtype == torch.bfloat16
    wide = torch.zeros(4, 264, device="cuda").half()
    for view in (wide[:, 4:260], wide[:, :256]):
        view.copy_(x)
        assert m._decoded_in_product(view) is None
        assert torch.allclose(m(view), y, rtol=1e-2, atol=1e-2)
    assert m(x[:0]).shape == (0, 64)


@pytest.mark.parametrize("kind", ["tensor", "parameter"])
def test_bias_and_scales_assigned_later(kind):
    """A bias given after construction, and scales that became a parameter, count for few tokens as for many."""
    wrap = (lambda t: torch.nn.Parameter(t, requires_grad=False)) if kind == "parameter" else (lambda t: t)
    m, w = layer(64, 256, 4, 64, False, False)
    bias = torch.linspace(-4, 4, 64).half()
    m.bias = wrap(bias.cuda())
    scales = m.scales
    del m.scales
    m.scales = wrap(scales)
    x = torch.randn(17, 256, generator=torch.Generator().manual_seed(3)).half()
    want = x.double() @ w.double().t() + bias.double()
    bound = 256 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t()) + 2.0 ** -11 * want.abs() + 2.0 ** -25
    for tokens in (4, 16, 17):
        assert (m._decoded_in_product(x[:tokens].cuda()) is not None) == (tokens <= 16)
        assert ((m(x[:tokens].cuda()).cpu().double() - want[:tokens]).abs() <= bound[:tokens]).all()


def test_trainable_bias_gets_its_gradient():
    m, _ = layer(64, 256, 4, 64, False, False)
    m.bias = torch.nn.Parameter(torch.zeros(64, device="cuda").half())
    for tokens in (4, 17):
        m.bias.grad = None
        m(torch.ones(tokens, 256, device="cuda").half()).sum().backward()
        assert torch.equal(m.bias.grad, torch.full_like(m.bias, tokens))
    with torch.no_grad():
        assert m._decoded_in_product(torch.ones(4, 256, device="cuda").half()) is not None


def test_one_group_without_g_idx():
    """dequantize_packed takes a missing g_idx as one group; so does the layer, for few tokens and many."""
    m, w = layer(64, 256, 4, -1, False, False)
    x = torch.randn(17, 256, generator=torch.Generator().manual_seed(4)).half()
    want = (x.double() @ w.double().t())
    m.g_idx = None
    for tokens in (4, 17):
        assert torch.allclose(m(x[:tokens].cuda()).cpu().double(), want[:tokens], rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("bits,d", [(4, 8), (4, 1048), (8, 72), (2, 80), (3, 96), (4, 4096)])
@pytest.mark.parametrize("act", [False, True])
def test_columns_behind_the_last_one_count_for_nothing(bits, d, act):
    """Codes equal to a large zero point: the weights are zero, the zero point alone times the scale is not finite."""
    from onecompression_b200.quantizer.gptq.gptq_layer import GPTQLinear

    out, top = 96, 2 ** bits - 1
    codes = torch.full((out, d), top, dtype=torch.int32)
    codes[1::2] -= torch.arange(d, dtype=torch.int32) % 2            # 0 and one negative step
    groups = (d + 31) // 32
    scale = torch.full((groups, out), 60000.0)
    zero = torch.full((groups, out), top, dtype=torch.int32)
    perm = torch.randperm(d, generator=torch.Generator().manual_seed(d)) if act else None
    m = GPTQLinear(d, out, bits, 32, act, codes, scale, zero, perm=perm)
    w = (60000.0 * (codes - top)).half()
    x = torch.randn(16, d, generator=torch.Generator().manual_seed(5)).mul(2.0 ** -14).half()
    want = x.double() @ w.double().t()
    bound = d * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t()) + 2.0 ** -11 * want.abs() + 2.0 ** -25
    for tokens in (1, 16):
        got = m._decoded_in_product(x[:tokens].cuda()).cpu().double()
        assert ((got - want[:tokens]).abs() <= bound[:tokens]).all()
