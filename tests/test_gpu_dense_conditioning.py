"""Backward stability of the dense Cholesky and its solve where the diagonal tiles themselves are ill-conditioned: the
residual of x, formed in extended precision, stays at rounding level whatever the condition of S.

Bound: the factorisation and two triangular solves by substitution satisfy (S + E) x = g with |E| <= gamma_{3n+1} |L| |L'|
(Higham, Accuracy and Stability of Numerical Algorithms, theorem 10.4); to first order, with || |L| |L'| || ~ ||S||, that is
||S x - g|| <= 3 n u ||S|| ||x||, u = 2^-53."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def kernel_matrix(n, cond):
    """Smooth in its indices, so that neighbouring rows (those of a tile) are nearly dependent."""
    i = np.arange(n)
    return np.exp(-(((i[:, None] - i[None, :]) / 8.0) ** 2)) + np.eye(n) * 20.0 / cond


def tile_matrix(n, cond):
    """L L' with the factors of its tiles ill-conditioned by their off-diagonal entries alone."""
    c = {1e8: -0.27, 1e10: -0.32, 1e12: -0.36}[cond]
    i = np.arange(n)
    L = np.where((i[:, None] // 64 == i[None, :] // 64) & (i[:, None] > i[None, :]), c, 0.0) + np.eye(n)
    return L @ L.T


@pytest.mark.parametrize("cond", [1e8, 1e10, 1e12])
@pytest.mark.parametrize("matrix", [kernel_matrix, tile_matrix])
@pytest.mark.parametrize("n", [60, 100, 300, 700])
def test_residual(bls, matrix, n, cond):
    S = matrix(n, cond)
    S = (S + S.T) / 2
    rng = np.random.default_rng(n)
    D = bls.DenseCholesky(n)
    assert D.factor(torch.from_numpy(np.triu(S).ravel(order="F")).to("cuda"))
    for g in (S @ rng.standard_normal(n), rng.standard_normal(n)):
        x = D.solve(torch.from_numpy(g).to("cuda")).cpu().numpy()
        r = S.astype(np.longdouble) @ x.astype(np.longdouble) - g.astype(np.longdouble)
        bound = 3 * n * 2.0**-53 * np.linalg.norm(S, 2) * np.linalg.norm(x)
        assert np.linalg.norm(r.astype(np.float64)) <= bound
