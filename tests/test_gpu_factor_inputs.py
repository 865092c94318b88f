"""The factor with NaNs on the diagonal and act-order, and with an order that the caller brings."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def spd(n, seed=0):
    x = torch.randn(2 * n + 16, n, generator=torch.Generator().manual_seed(seed), dtype=torch.float64)
    h = (x.t() @ x / len(x)).float()
    return ((h + h.t()) / 2).to(DEV)


@pytest.mark.parametrize("n", [5, 130, 1300])
def test_nan_on_the_diagonal_leaves_a_permutation(n):
    from onecompression_b200 import kernels as K

    h = spd(n)
    bad = [1, n // 2, n - 1]
    for j in bad:
        h[j, j] = float("nan")
    two = K.factor_hessians_batched(torch.stack([h, spd(n)]), 0.01, True)
    perm = two["perm"].cpu()
    iota = torch.arange(n, dtype=torch.int32)
    assert torch.equal(perm.sort(1).values, iota.expand(2, -1))
    assert perm[0, :3].tolist() == bad
    for b in range(2):
        assert torch.equal(two["invperm"][b].cpu()[perm[b].long()], iota)
    status = two["status"].cpu()
    assert status[0] > 0 and status[1] == 0
    with pytest.raises(RuntimeError, match="Cholesky"):
        K.factor_hessian(h, 0.01, True)


def hinv_factor(h, perm, invperm, actorder, reuse_perm, workspace=None):
    """(u, status) of the C entry point."""
    from onecompression_b200 import _lib
    from onecompression_b200._lib import call, ptr, stream_handle

    n = len(h)
    u = torch.empty(n, n, device=DEV)
    dead = torch.empty(n, dtype=torch.uint8, device=DEV)
    damp, status = torch.empty(2, device=DEV), torch.empty(1, dtype=torch.int32, device=DEV)
    if workspace is None:
        workspace = torch.empty(_lib.load().oc_hinv_workspace_bytes(n), dtype=torch.uint8, device=DEV)
    call("oc_hinv_factor", ptr(h), n, n, 0.01, 1.0, actorder, reuse_perm, ptr(u), n, ptr(perm), ptr(invperm), ptr(dead),
         ptr(damp), ptr(status), ptr(workspace), workspace.numel(), stream_handle())
    return u, int(status.item())


@pytest.mark.parametrize("n", [4, 65, 130, 516])
@pytest.mark.parametrize("actorder", [0, 1])
def test_reuse_perm_takes_the_callers_order(n, actorder):
    h = spd(n)
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(n)).to(torch.int32).to(DEV)
    invperm = torch.argsort(perm.long()).int()
    kept = perm.clone(), invperm.clone()
    u, status = hinv_factor(h, perm, invperm, actorder, 1)
    p = perm.long()
    want, want_status = hinv_factor(h[p][:, p].contiguous(), torch.empty_like(perm), torch.empty_like(perm), 0, 0)
    assert status == want_status == 0 and torch.equal(u, want)
    assert torch.equal(perm, kept[0]) and torch.equal(invperm, kept[1])
