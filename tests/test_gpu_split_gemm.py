"""Products of operands split into two scaled fp16 planes (oc_gemm_split_f32), against float64."""

import pytest
import torch

from onecompression_b200 import kernels as K

pytestmark = pytest.mark.gpu
SKIP_UPPER, KLO_N, KHI_M, KHI_N, KLO_M = 1, 2, 4, 8, 16


def rnd(*shape, seed=0, spread=0.0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(*shape, generator=g)
    if spread:
        x *= torch.exp2(spread * torch.rand(shape[0], 1, generator=g))
    return x.cuda()


def bound(a, b, k):
    """Row and column norms bound an entry of the product; each product is off by 2 * 2^-23 + 2^-22 at most,
    each of the k / 16 accumulations of a chain of 128 (three a step) by 2^-23 of the partial sum, the sum over
    chains by 2^-24 per chain: below 2^-18 in all for the sizes here."""
    return a.norm(dim=1)[:, None] * b.norm(dim=0)[None, :] * 2.0**-18


def check(got, a, b, c0, alpha):
    a64, b64 = a.double(), b.double()
    want = alpha * (a64 @ b64) + (c0.double() if c0 is not None else 0)
    lim = abs(alpha) * bound(a64, b64, a.shape[1]) + 2.0**-22 * want.abs() + 1e-30
    assert ((got.double() - want).abs() <= lim).all(), ((got.double() - want).abs() / lim).max().item()
    assert K.gemm_tc_status() == 0


@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("m,n,k", [(128, 128, 128), (1, 1, 1), (129, 257, 33), (300, 200, 160), (64, 640, 15),
                                   (256, 128, 384), (1000, 520, 700), (127, 255, 129)])
@pytest.mark.parametrize("add", [False, True])
def test_layouts_and_ragged_sizes(ta, tb, m, n, k, add):
    a, b = rnd(m, k, seed=1), rnd(k, n, seed=2)
    n4 = (n + 3) // 4 * 4          # (rows are written in whole groups of four)
    out = {}
    for shape in (1, 2, 0):
        c = rnd(m, n4 + 4, seed=3)
        c0 = c.clone()
        old = K.set_gemm_tile_shape(shape)
        try:
            K.gemm_split(a.t().contiguous() if ta else a, b.t().contiguous() if tb else b, c[:, :n], alpha=-1.5,
                         add=add, trans_a=ta, trans_b=tb)
        finally:
            K.set_gemm_tile_shape(old)
        assert torch.equal(c[:, n4:], c0[:, n4:])
        out[shape] = c[:, :n]
    check(out[0], a, b, c0[:, :n] if add else None, -1.5)
    assert torch.equal(out[1], out[2]) and torch.equal(out[1], out[0])


@pytest.mark.parametrize("rows_scaled", [False, True])
@pytest.mark.parametrize("spread", [0.0, 14.0])
def test_rows_of_different_size(rows_scaled, spread):
    a, b = rnd(520, 390, seed=4, spread=spread), rnd(390, 300, seed=5)
    got = K.gemm_split(a, b, rows_scaled=rows_scaled)
    check(got, a, b, None, 1.0)


def test_scaled_rows_do_not_depend_on_their_neighbours():
    a, b = rnd(256, 256, seed=6, spread=30.0), rnd(256, 256, seed=7)
    a[5] = float("inf")
    a[9, 3] = float("nan")
    a[17] = 0
    a[33] *= 1e-30
    whole = K.gemm_split(a, b, rows_scaled=True)
    assert whole[9].isnan().all() and not whole[5].isfinite().any() and (whole[17] == 0).all()
    for r in (0, 4, 6, 33, 100, 255):
        alone = K.gemm_split(a[r:r + 1].contiguous(), b, rows_scaled=True)
        assert torch.equal(whole[r], alone[0]) and alone.isfinite().all()


@pytest.mark.parametrize("flag", [KLO_N, KHI_M, KHI_N, KLO_M])
@pytest.mark.parametrize("n", [640, 1000])
def test_triangular_ranges(flag, n):
    other, tri = rnd(n, n, seed=8), rnd(n, n, seed=9)
    tri = {KLO_N: tri.tril(), KHI_M: tri.tril(), KHI_N: tri.triu(), KLO_M: tri.triu()}[flag].contiguous()
    a, b = (tri, other) if flag in (KHI_M, KLO_M) else (other, tri)
    out = {}
    for shape in (1, 2):
        old = K.set_gemm_tile_shape(shape)
        try:
            out[shape] = K.gemm_split(a, b, flags=flag)
        finally:
            K.set_gemm_tile_shape(old)
    check(out[1], a, b, None, 1.0)
    assert torch.equal(out[1], out[2])


@pytest.mark.parametrize("m,n,k", [(640, 640, 512), (2900, 2900, 128), (1300, 384, 128), (130, 130, 64)])
def test_lower_tiles_only(m, n, k):
    p = rnd(m, k, seed=10)
    out = {}
    for shape in (1, 2):
        old = K.set_gemm_tile_shape(shape)
        c0 = rnd(m, (n + 3) // 4 * 4, seed=11)[:, :n]
        out[shape] = c0.clone() if n % 4 == 0 else torch.empty_strided(c0.shape, c0.stride(), device="cuda").copy_(c0)
        try:
            K.gemm_split(p, p[:n].contiguous(), out[shape], alpha=-1.0, add=True, trans_b=True, flags=SKIP_UPPER)
        finally:
            K.set_gemm_tile_shape(old)
    assert torch.equal(out[1], out[2])
    tile = torch.arange(m, device="cuda")[:, None] // 128 >= torch.arange(n, device="cuda")[None, :] // 128
    want = c0.double() - p.double() @ p[:n].double().t()
    lim = bound(p.double(), p[:n].double().t(), k) + 2.0**-22 * want.abs()
    assert ((out[1].double() - want).abs() <= lim)[tile].all()
    assert torch.equal(out[1][~tile], c0[~tile])
    assert K.gemm_tc_status() == 0
