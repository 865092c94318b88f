"""Decoding of the packed layout, against the formula in float64 rounded once: groups that end inside eight columns,
single columns behind the last whole eight, orders with and without runs, an index that does not lie at 16 bytes."""

import pytest
import torch

from onecompression_b200 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["runs", "one group", "permuted", "reversed", "shifted"])
@pytest.mark.parametrize("bits,out,d,gs", [(4, 64, 256, 128), (4, 200, 1000, 40), (4, 8, 8, 4), (8, 36, 260, 20), (8, 64, 132, 64),
                                           (2, 80, 304, 32), (2, 16, 144, 12), (3, 96, 352, 32), (3, 32, 32, 5)])
def test_dequantize(bits, out, d, gs, order):
    g = torch.Generator(device="cuda").manual_seed(bits * d)
    groups = 1 if order == "one group" else -(-d // gs)
    codes = torch.randint(0, 1 << bits, (out, d), generator=g, device="cuda", dtype=torch.int32)
    zeros = torch.randint(1, 1 << bits, (groups, out), generator=g, device="cuda", dtype=torch.int32)
    scales = (torch.rand(groups, out, generator=g, device="cuda") * 0.02).half()
    scales[0, 0] = 60000.0        # (overflows)
    scales[0, 1] = 6e-8           # (subnormal)
    idx = (torch.arange(d, device="cuda") // gs if groups > 1 else torch.zeros(d, device="cuda")).int()
    if order == "permuted":
        idx = idx[torch.randperm(d, generator=g, device="cuda")].contiguous()
    elif order == "reversed":
        idx = idx.flip(0).contiguous()
    elif order == "shifted":
        idx = torch.cat([idx[:1], idx])[1:]
        assert idx.data_ptr() % 16
    got = K.dequantize_packed(K.pack_qweight(codes, bits), K.pack_qzeros(zeros, bits, add=-1), scales, idx, bits, (out, d))
    z = zeros[idx.long()].t().double()
    want = (scales[idx.long()].t().double() * (codes.double() - z)).half()
    assert torch.equal(got, want)
