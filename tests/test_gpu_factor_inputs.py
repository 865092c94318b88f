"""Inputs of the factor that are no ordinary Hessian: NaNs on the diagonal with act-order."""

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
