"""The dense Cholesky and its one-launch solve at the edges of their schedule: 64-column tiles, groups of four of them, the
identity padding, a pivot that fails in each part of it, x in the place of g, repeated solves. Tolerance 1e-10 relative, as
in test_gpu_dense.py: random systems of condition below 1e3, FP64 throughout."""
import numpy as np
import pytest
import torch

from test_gpu_dense import first_bad_pivot, relerr

pytestmark = pytest.mark.gpu


def spd(n, seed):
    rng = np.random.default_rng(seed)
    B = rng.standard_normal((n, n))
    return B @ B.T / n + np.eye(n), rng


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("n", [2, 191, 192, 193, 255, 256, 257, 319, 320, 321, 385, 577, 1025])
def test_tiles_and_groups(bls, n, dtype):
    A, rng = spd(n, n)
    A = A.astype(np.float32).astype(np.float64) if dtype == torch.float32 else A
    D = bls.DenseCholesky(n)
    S = torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda", dtype)
    assert D.factor(S)
    for k in range(2):
        g = rng.standard_normal(n)
        x = torch.from_numpy(g).to("cuda")
        assert D.solve(x, x) is x   # in place
        assert relerr(x.cpu().numpy(), np.linalg.solve(A, g)) <= 1e-10
    s_r = 0.5 + rng.random(n)
    assert D.factor(S, 0.25, torch.from_numpy(s_r).to("cuda"))
    x = D.solve(torch.from_numpy(g).to("cuda"))
    assert relerr(x.cpu().numpy(), np.linalg.solve(A + 0.25 * np.diag(s_r), g)) <= 1e-10


@pytest.mark.parametrize("column", [1, 16, 17, 64, 65, 128, 200, 256, 257, 320, 321, 400])
def test_failing_pivot(bls, column):
    n = 400
    A, _ = spd(n, 7)
    A[column - 1, column - 1] = -5.0
    assert first_bad_pivot(A) == column
    D = bls.DenseCholesky(n)
    S = torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda")
    assert not D.factor(S) and D.failed_column == column
    with pytest.raises(bls.ArgumentError):
        D.solve(torch.zeros(n, dtype=torch.float64, device="cuda"))
    A[column - 1, column - 1] = 5.0
    assert D.factor(torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda")) and D.failed_column == 0


def test_non_finite_right_hand_side(bls):
    """A NaN of any payload in g passes through the solve (its exchange marks unwritten values by a payload of its own)."""
    n = 200
    A, rng = spd(n, 3)
    D = bls.DenseCholesky(n)
    assert D.factor(torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda"))
    g = rng.standard_normal(n)
    g[150:] = np.frombuffer(b"\xff" * 8, np.float64)[0]
    x = D.solve(torch.from_numpy(g).to("cuda")).cpu().numpy()
    assert np.isnan(x).all()
