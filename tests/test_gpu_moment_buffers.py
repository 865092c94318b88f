"""Moments into buffers that were not cleared: odd widths on both engines, no tokens at all, mirrored lower part."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [8, 60, 64, 72, 200, 264, 1000, 57])
@pytest.mark.parametrize("cross", [False, True])
@pytest.mark.parametrize("chunks", [(), (1,), (700,), (64, 0, 129)])
def test_moments_do_not_read_what_was_there(d, cross, chunks):
    from onecompression_b200 import kernels as K

    dev = torch.device("cuda:0")
    # leave NaNs where the accumulator is going to be allocated
    junk = [torch.full((d, d), float("nan"), device=dev) for _ in range(3)]
    del junk
    g = torch.Generator().manual_seed(d)
    acc = K.MomentAccumulator(d, dev, cross=cross)
    xs = [(torch.randn(t, d, generator=g).half(), torch.randn(t, d, generator=g).half()) for t in chunks]
    for xq, xf in xs:
        acc.add(xq.to(dev), xf.to(dev) if cross else None)
    h, c, n = acc.finalize()
    assert n == sum(chunks)
    xq = torch.cat([x for x, _ in xs] + [torch.zeros(0, d).half()]).double()
    xf = torch.cat([x for _, x in xs] + [torch.zeros(0, d).half()]).double()
    want = 2 / max(n, 1) * xq.t() @ xq
    if acc.force_simt:
        # (slices of 256 tokens are added atomically, in any order: a rounding each of at most two partial sums)
        assert (h - h.t()).abs().max() <= 4 * 2.0 ** -24 * h.abs().max() * 2
    else:
        assert torch.equal(h, h.t())
    # sums of n products in fp32 and truncating tensor-core chains of at most 512 tokens
    bound = 1e-5 * max(1.0, float(want.abs().max()))
    assert (h.cpu().double() - want).abs().max() <= bound
    if cross:
        want = 2 / max(n, 1) * (xf - xq).t() @ xq
        assert (c.cpu().double() - want).abs().max() <= 1e-5 * max(1.0, float(want.abs().max()))
    fresh = K.MomentAccumulator(d, dev, cross=cross)
    assert not fresh.H.any() and (fresh.C is None or not fresh.C.any())


@pytest.mark.parametrize("n,pad", [(1, 0), (3, 1), (64, 0), (65, 3), (130, 2), (1000, 0), (1000, 1)])
def test_mirror(n, pad):
    from onecompression_b200._lib import call, ptr, stream_handle

    m = torch.randn(n, n + pad, device="cuda")
    want = m.clone()
    want[:, :n] = torch.triu(m[:, :n]) + torch.triu(m[:, :n], 1).t()
    call("oc_mirror_upper", ptr(m), n + pad, n, stream_handle())
    assert torch.equal(m, want)


def chunk(t, d, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(t, d, generator=g).half().cuda(), torch.randn(t, d, generator=g).half().cuda()


def same(got, want):
    return torch.allclose(got, want, rtol=0, atol=1e-5 * max(1.0, float(want.abs().max())))


@pytest.mark.parametrize("d", [57, 264])
def test_moments_are_saved_and_put_back(d):
    """H, C and nsamples of one accumulator, assigned to another that goes on, or added to its own."""
    from onecompression_b200 import kernels as K

    (q0, f0), (q1, f1) = chunk(100, d, 0), chunk(60, d, 1)
    whole, first = K.MomentAccumulator(d, "cuda", cross=True), K.MomentAccumulator(d, "cuda", cross=True)
    whole.add(q0, f0)
    whole.add(q1, f1)
    first.add(q0, f0)
    saved = [t.clone() for t in first.finalize()[:2]]
    junk = [torch.full((d, d), float("nan"), device="cuda") for _ in range(3)]
    del junk
    rest = K.MomentAccumulator(d, "cuda", cross=True)
    rest.H, rest.C, rest.nsamples = saved[0], saved[1], 100
    rest.add(q1, f1)
    h, c, n = whole.finalize()
    h2, c2, n2 = rest.finalize()
    assert n2 == n and same(h2, h) and same(c2, c)
    # what one of the two assignments leaves out is zero
    junk = torch.full((d, d), float("nan"), device="cuda")
    del junk
    half = K.MomentAccumulator(d, "cuda", cross=True)
    half.H = torch.eye(d, device="cuda")
    assert torch.equal(half.H, torch.eye(d, device="cuda")) and not half.C.any()
    half.C += 2
    half.H *= 3
    assert torch.equal(half.H, 3 * torch.eye(d, device="cuda")) and bool((half.C == 2).all())


@pytest.mark.parametrize("d", [57, 264])
def test_an_add_that_failed_counts_for_nothing(d, monkeypatch):
    """No memory for the scratch, then a launch that is refused: the next chunk is the first one."""
    from onecompression_b200 import kernels as K

    q, f = chunk(64, d, 2)
    want = K.MomentAccumulator(d, "cuda", cross=True)
    want.add(q, f)
    junk = [torch.full((d, d), float("nan"), device="cuda") for _ in range(3)]
    del junk
    acc = K.MomentAccumulator(d, "cuda", cross=True)

    def refuse(*args, **kwargs):
        raise RuntimeError("refused")

    for name, holder in (("empty", torch), ("call", K)):
        if name == "empty" and d % 8:
            continue                     # the FMA engine needs no scratch
        with monkeypatch.context() as m:
            m.setattr(holder, name, refuse)
            with pytest.raises(RuntimeError, match="refused"):
                acc.add(torch.cat([q, q]), torch.cat([f, f]))
        assert acc.nsamples == 0
    acc.add(q, f)
    for got, ref in zip(acc.finalize()[:2], want.finalize()[:2]):
        assert torch.equal(got, ref)


@pytest.mark.parametrize("d", [57, 264])
def test_a_sample_count_set_from_outside_weighs_zeros(d):
    from onecompression_b200 import kernels as K

    q, f = chunk(64, d, 3)
    want = K.MomentAccumulator(d, "cuda", cross=True)
    want.add(q, f)
    junk = [torch.full((d, d), float("nan"), device="cuda") for _ in range(3)]
    del junk
    acc = K.MomentAccumulator(d, "cuda", cross=True)
    acc.nsamples = 64
    acc.add(q, f)
    for got, ref in zip(acc.finalize()[:2], want.finalize()[:2]):
        assert same(2 * got, ref)


@pytest.mark.parametrize("d", [57, 264, 1000])
def test_h_between_two_chunks(d):
    """Both triangles, whatever was in memory; reading it changes nothing of what comes out in the end."""
    from onecompression_b200 import kernels as K

    (q0, _), (q1, _) = chunk(100, d, 4), chunk(60, d, 5)
    want = K.MomentAccumulator(d, "cuda")
    want.add(q0)
    after_one = K.MomentAccumulator(d, "cuda")
    after_one.add(q0)
    want.add(q1)
    junk = [torch.full((d, d), float("nan"), device="cuda") for _ in range(3)]
    del junk
    acc = K.MomentAccumulator(d, "cuda")
    acc.add(q0)
    assert torch.equal(acc.H, after_one.finalize()[0]) and torch.equal(acc.H, acc.H.t())
    acc.add(q1)
    assert torch.equal(acc.H, acc.H.t())
    assert torch.equal(acc.finalize()[0], want.finalize()[0])
