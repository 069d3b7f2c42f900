"""A pivot that fails while panels and updates of the same factorisation run beside it, on other streams: the kernels that
read the failure word decide for a whole CTA at once, the failing column is the first one, and the solver is usable
afterwards. Tolerance 1e-10 relative as in test_gpu_dense.py."""
import numpy as np
import pytest
import torch

from test_gpu_dense import relerr
from test_gpu_dense_tiles import spd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [130, 700, 1500])
def test_failure_beside_running_updates(bls, n):
    A, rng = spd(n, 11)
    D = bls.DenseCholesky(n)
    S = torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda").view(n, n)
    diag = torch.diagonal(S)
    g = rng.standard_normal(n)
    for column in sorted(rng.choice(n, 40, replace=False)):
        good = diag[column].item()
        diag[column] = -5.0
        assert not D.factor(S.view(-1)) and D.failed_column == column + 1
        diag[column] = good
        assert D.factor(S.view(-1)) and D.failed_column == 0
        x = D.solve(torch.from_numpy(g).to("cuda"))
    assert relerr(x.cpu().numpy(), np.linalg.solve(A, g)) <= 1e-10


def test_a_wait_that_gives_up_is_reported(bls):
    """With one poll allowed per wait the later tiles cannot have the first one's values: the solve ends, its x is marked
    by NaNs, and the next synchronising call raises, once. The solver goes on working."""
    n = 640
    A, rng = spd(n, 5)
    D = bls.DenseCholesky(n)
    S = torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda")
    g = rng.standard_normal(n)
    want = np.linalg.solve(A, g)
    limit = bls._lib.gpu().bls_dense_solver_set_wait_limit
    assert limit(D.handle, 0) == bls._lib.BLS_EINVAL
    assert D.factor(S)
    for report in (D.check, lambda: D.factor(S)):
        assert limit(D.handle, 1) == 0
        x = D.solve(torch.from_numpy(g).to("cuda"))
        assert torch.isnan(x).any()
        with pytest.raises(bls.BlsError, match="wait"):
            report()
        D.check()
        assert limit(D.handle, 1 << 22) == 0
        x = D.solve(torch.from_numpy(g).to("cuda"))
        D.check()
        assert relerr(x.cpu().numpy(), want) <= 1e-10
    assert D.factor(S) and D.failed_column == 0


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33, 48, 49, 65, 80, 81, 96, 97, 113, 127])
def test_padding_in_the_last_tile(bls, n):
    """The last tile's padding is left out in steps of 16 columns, and its inverse is formed with it."""
    A, rng = spd(n, n + 1)
    D = bls.DenseCholesky(n)
    S = torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda")
    for _ in range(2):
        assert D.factor(S)
        g = rng.standard_normal(n)
        assert relerr(D.solve(torch.from_numpy(g).to("cuda")).cpu().numpy(), np.linalg.solve(A, g)) <= 1e-10
    A[n - 1, n - 1] = -1.0
    assert not D.factor(torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda")) and D.failed_column == n
