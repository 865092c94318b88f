"""Which operands the packed layer's one-kernel path takes, and when it leaves a call to the general path.
The kernels are replaced by the same sums in torch."""

import pytest
import torch

from onecompression_b200 import _lib, kernels
from onecompression_b200.quantizer.gptq import gptq_layer
from onecompression_b200.quantizer.gptq.gptq_layer import GPTQLinear

OUT, D = 8, 16


def decoded(qweight, qzeros, scales, g_idx, wbits, shape):
    assert wbits == 4
    nibble = 4 * torch.arange(8, dtype=torch.int32)
    q = ((qweight[:, None, :] >> nibble[None, :, None]) & 15).reshape(shape[1], shape[0])
    z = (((qzeros[:, :, None] >> nibble) & 15).reshape(-1, shape[0]) + 1) & 15
    g = g_idx.long()
    return (scales[g].float() * (q - z[g]).float()).t().half()


@pytest.fixture
def calls(monkeypatch):
    seen = []

    def packed_linear(x, qweight, qzeros, scales, g_idx, bias, wbits, out, d):
        if x.numel() // d > kernels.PACKED_LINEAR_TOKENS:
            return None
        seen.append((qweight, qzeros, scales, g_idx, bias))
        y = x.float() @ decoded(qweight, qzeros, scales, g_idx, wbits, (out, d)).float().t()
        return (y if bias is None else y + bias.float()).half().detach()

    monkeypatch.setattr(kernels, "packed_linear", packed_linear)
    monkeypatch.setattr(kernels, "dequantize_packed", decoded)
    return seen


def layer(bias=None):
    g = torch.Generator().manual_seed(1)
    word = lambda *shape: torch.randint(-2 ** 31, 2 ** 31 - 1, shape, generator=g, dtype=torch.int64).int()
    return GPTQLinear(D, OUT, 4, 8, False, word(D // 8, OUT), torch.rand(2, OUT, generator=g).half() * 0.1,
                      word(2, OUT // 8), bias=bias, device="cpu", input_weight_is_packed=True,
                      input_zero_is_packed=True)


def check(m, calls, short=True):
    """The first four of 17 tokens, alone and in the long call (which takes the general path)."""
    x = torch.randn(17, D, generator=torch.Generator().manual_seed(2)).half()
    before = len(calls)
    got = m(x[:4])
    assert len(calls) == before + (1 if short else 0)
    want = m(x)[:4]
    assert len(calls) == before + (1 if short else 0)
    assert torch.allclose(got, want, rtol=2e-3, atol=2e-3)
    return got


BIAS = torch.linspace(-3, 3, OUT).half()


@pytest.mark.parametrize("built_with", [None, torch.zeros(OUT)])
@pytest.mark.parametrize("assigned", ["tensor", "parameter", "none"])
def test_bias_assigned_after_construction(calls, built_with, assigned):
    m = layer(built_with)
    plain = check(layer(), calls)
    m.bias = {"tensor": BIAS, "parameter": torch.nn.Parameter(BIAS, requires_grad=False), "none": None}[assigned]
    got = check(m, calls)
    assert torch.allclose(got - plain, torch.zeros(OUT).half() if assigned == "none" else BIAS, atol=5e-3)


@pytest.mark.parametrize("name", ["qweight", "qzeros", "scales", "g_idx"])
def test_operand_replaced_by_a_parameter_or_a_plain_attribute(calls, name):
    want = check(layer(), calls)
    m = layer()
    t = getattr(m, name)
    delattr(m, name)
    m.register_parameter(name, torch.nn.Parameter(t, requires_grad=False))
    assert torch.equal(check(m, calls), want) and calls[-1][["qweight", "qzeros", "scales", "g_idx"].index(name)] is getattr(m, name)
    m = layer()
    delattr(m, name)
    setattr(m, name, t)
    assert torch.equal(check(m, calls), want)


@pytest.mark.parametrize("name", ["bias", "scales"])
def test_trainable_operands_keep_the_general_path(calls, name):
    m = layer(BIAS)
    t = getattr(m, name)
    delattr(m, name)
    m.register_parameter(name, torch.nn.Parameter(t))
    x = torch.ones(4, D).half()
    with torch.no_grad():
        want = check(m, calls)                       # no graph to build: one kernel
    assert torch.allclose(check(m, calls, short=False), want, rtol=2e-3, atol=2e-3)
    m(x).sum().backward()
    if name == "bias":
        assert torch.equal(m.bias.grad, torch.full((OUT,), 4.0).half())
    m.requires_grad_(False)
    assert torch.equal(check(m, calls), want)


def test_a_decoding_of_its_own_is_used_for_a_few_tokens_too(calls):
    class Doubled(GPTQLinear):
        def dequantized_weight(self):
            return 2 * super().dequantized_weight()

    m = layer()
    plain = check(m, calls)
    m.__class__ = Doubled
    assert torch.allclose(check(m, calls, short=False), 2 * plain, rtol=2e-3, atol=2e-3)
    m = layer()
    original = m.dequantized_weight
    m.dequantized_weight = lambda: 3 * original()
    assert torch.allclose(check(m, calls, short=False), 3 * plain, rtol=2e-3, atol=2e-3)


def test_the_kernel_is_not_offered_a_layer_without_g_idx():
    class OnGpu:                  # what packed_linear asks of its input before it looks at the operands
        dtype, is_cuda, shape = torch.float16, True, torch.Size([4, D])
        dim = lambda self: 2
        is_contiguous = lambda self: True
        numel = lambda self: 4 * D
        get_device = lambda self: 0

    m = layer()
    assert kernels.packed_linear(OnGpu(), m.qweight, m.qzeros, m.scales, None, None, 4, OUT, D) is None


@pytest.mark.parametrize("holder,name", [(torch._C, "_len_torch_function_stack"), (torch._C, "_len_torch_dispatch_stack"),
                                         (torch._C._functorch, "peek_interpreter_stack"),
                                         (torch.autograd.forward_ad, "_current_level")])
def test_a_torch_without_an_internal_name_has_the_general_path(calls, monkeypatch, holder, name):
    with monkeypatch.context() as m:
        m.delattr(holder, name)
        found = gptq_layer._watchers()
    assert found is None
    monkeypatch.setattr(gptq_layer, "_WATCHERS", found)
    check(layer(), calls, short=False)


def test_stream_handle_without_the_internal_name(monkeypatch):
    class Stream:
        def __init__(self, index):
            self.cuda_stream = 7 + index

    monkeypatch.setattr(torch.cuda, "current_stream", Stream)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    monkeypatch.setattr(_lib, "_raw_stream", None)
    assert _lib.stream_handle() == 8 and _lib.stream_handle(2) == 9


def test_compiled_layer(calls):
    """A compiler sees the general path."""
    m = layer(BIAS)
    x = torch.randn(4, D, generator=torch.Generator().manual_seed(2)).half()
    want = m(x)
    before = len(calls)
    got = torch.compile(m, backend="eager")(x)
    assert len(calls) == before and torch.allclose(got, want, rtol=2e-3, atol=2e-3)
