"""Workspaces that start 4 or 8 bytes behind a 16-byte boundary: the results are those of an aligned one."""

import pytest
import torch

from test_gpu_factor_inputs import hinv_factor, spd

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.fixture
def fma_engine():
    """Products on the FMA engine, which takes every alignment with the same arithmetic."""
    from onecompression_b200 import _lib

    old = _lib.load().oc_set_gemm_engine(1)
    yield
    _lib.load().oc_set_gemm_engine(old)


@pytest.fixture
def workspace_at(monkeypatch):
    """Makes the wrappers' workspaces start ``offset`` bytes behind a 256-byte boundary."""
    from onecompression_b200 import kernels as K

    def at(offset):
        monkeypatch.setattr(K, "_workspace", lambda nbytes, device: torch.full(
            (nbytes + 256,), 0xff, dtype=torch.uint8, device=device)[offset:offset + nbytes])

    return at


@pytest.mark.parametrize("out,d,gs,act", [(40, 64, 32, False), (300, 264, 24, True), (70, 520, -1, True), (64, 128, 128, False)])
def test_column_loop(fma_engine, workspace_at, out, d, gs, act):
    from onecompression_b200 import kernels as K

    f = K.factor_hessian(spd(d), 0.01, act)
    w = torch.randn(out, d, generator=torch.Generator().manual_seed(out)).mul(0.02).half().to(DEV)
    results = []
    for offset in (0, 4, 8):
        workspace_at(offset)
        results.append(K.gptq_quantize(w, f, 4, gs, False, pack=False, want_codes=True, want_scales_f32=True))
    for r in results[1:]:
        assert all(torch.equal(r[k], results[0][k]) for k in r)


@pytest.mark.parametrize("out,d,act", [(33, 64, False), (40, 260, True)])
def test_correction(fma_engine, workspace_at, out, d, act):
    from onecompression_b200 import kernels as K

    f = K.factor_hessian(spd(d), 0.01, act)
    g = torch.Generator().manual_seed(out)
    w = torch.randn(out, d, generator=g).mul(0.02).half().to(DEV)
    c = (0.05 * torch.randn(d, d, generator=g)).to(DEV)
    results = []
    for offset in (0, 4, 8):
        workspace_at(offset)
        results.append(w.clone())
        K.qep_adjust(results[-1], c, f, 0.5)
    assert torch.equal(results[1], results[0]) and torch.equal(results[2], results[0])


@pytest.mark.parametrize("n", [4, 64, 124, 127])
def test_factor(n):
    from onecompression_b200 import _lib

    h = spd(n)
    nbytes = _lib.load().oc_hinv_workspace_bytes(n)
    perm = torch.empty(n, dtype=torch.int32, device=DEV)
    results = []
    for offset in (0, 4, 8):
        ws = torch.full((nbytes + 256,), 0xff, dtype=torch.uint8, device=DEV)[offset:offset + nbytes]
        u, status = hinv_factor(h, perm, perm.clone(), 1, 0, ws)
        assert status == 0
        results.append(u)
    assert torch.equal(results[1], results[0]) and torch.equal(results[2], results[0])


def test_factor_of_full_panels_wants_16_bytes():
    from onecompression_b200 import _lib

    n = 128
    nbytes = _lib.load().oc_hinv_workspace_bytes(n)
    ws = torch.empty(nbytes + 256, dtype=torch.uint8, device=DEV)
    perm = torch.empty(n, dtype=torch.int32, device=DEV)
    with pytest.raises(_lib.KernelError, match="16-byte aligned"):
        hinv_factor(spd(n), perm, perm.clone(), 0, 0, ws[4:4 + nbytes])


@pytest.mark.parametrize("n", [130, 516, 1160])
def test_factor_does_not_read_what_was_there(n):
    from onecompression_b200 import _lib

    h = spd(n)
    perm = torch.empty(n, dtype=torch.int32, device=DEV)
    u = [hinv_factor(h, perm, perm.clone(), 1, 0, torch.full((_lib.load().oc_hinv_workspace_bytes(n),), fill,
                                                             dtype=torch.uint8, device=DEV))[0] for fill in (0, 0xff)]
    assert torch.equal(u[0], u[1])
