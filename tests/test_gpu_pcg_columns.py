"""The one-launch PCG on patterns of 6-column blocks, against a dense FP64 solve of the same stored S, where its shares of
the columns and its windows can go wrong: one camera, fewer blocks than warps, a window wider than the shared-memory one
(every camera coupled to every other), warm starts, an iteration limit, g = 0, and an S that cannot be read in pairs.

The solution's tolerance follows from the stopping rule: ||x - x*|| <= cond(S) tol ||x*||, cond(S) below 50 by
construction (diagonally dominant blocks), tol = 1e-10."""
import numpy as np
import pytest
import torch

from test_gpu_column_runs import couplings
from test_gpu_schur import cu, relerr

pytestmark = pytest.mark.gpu


def system(bls, ncam, npts, kmax, seed, dtype=np.float64):
    """A random symmetric S on the pattern of a scene, diagonally dominant: (structure, pattern, nzval, dense S)."""
    rng = np.random.default_rng(seed)
    st = bls.SchurStructure.positional([6] * ncam, [3] * npts, couplings(rng, ncam, npts, 1, kmax))
    pat = bls.build_schur_pattern(st)
    nz = rng.uniform(-1, 1, pat.nnz)
    col = np.repeat(np.arange(st.nr), np.diff(pat.S_colptr))
    A = np.zeros((st.nr, st.nr))
    up = pat.S_rowval <= col
    A[pat.S_rowval[up], col[up]] = nz[up]
    A = np.triu(A, 1) + np.triu(A, 1).T
    nz[pat.diag_inds] = np.abs(A).sum(1).max() * (1.05 + 0.2 * rng.random(st.nr))
    nz = nz.astype(dtype)
    A[np.arange(st.nr), np.arange(st.nr)] = 0
    B = np.zeros_like(A)
    B[pat.S_rowval[up], col[up]] = nz[up].astype(np.float64)
    return st, pat, nz, np.triu(B) + np.triu(B, 1).T


CASES = [(1, 4, 1), (2, 9, 2), (7, 40, 4), (33, 300, 6), (190, 900, 30), (260, 40, 250), (401, 3000, 5)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("ncam,npts,kmax", CASES)
def test_against_dense_solve(bls, ncam, npts, kmax, dtype):
    st, pat, nz, A = system(bls, ncam, npts, kmax, ncam, dtype)
    rng = np.random.default_rng(1)
    g = rng.standard_normal(st.nr)
    ws = bls.PCGWorkspace(st, pat)
    want = np.linalg.solve(A, g)
    x, res = ws.solve(cu(nz), cu(g), tol=1e-10)
    assert res.converged and res.rel_residual <= 1e-10
    assert relerr(x.cpu().numpy(), want) <= 50 * 1e-10
    # from the solution: nothing to do; from elsewhere: the same solution
    again, res = ws.solve(cu(nz), cu(g), x.clone(), tol=1e-9)
    assert res.converged and res.iterations == 0 and torch.equal(again, x)
    y, res = ws.solve(cu(nz), cu(g), cu(rng.standard_normal(st.nr)), tol=1e-10)
    assert res.converged and relerr(y.cpu().numpy(), want) <= 50 * 1e-10
    # S one entry past its alignment: the form of separate launches
    buf = torch.zeros(len(nz) + 1, dtype=torch.float64 if dtype == np.float64 else torch.float32, device="cuda")
    buf[1:] = cu(nz)
    z, res = ws.solve(buf[1:], cu(g), tol=1e-10)
    assert res.converged and relerr(z.cpu().numpy(), want) <= 50 * 1e-10


def test_limit_zero_and_failure(bls):
    st, pat, nz, A = system(bls, 40, 400, 5, 3)
    g = np.random.default_rng(2).standard_normal(st.nr)
    ws = bls.PCGWorkspace(st, pat)
    x, res = ws.solve(cu(nz), cu(g), tol=1e-14, maxit=2)
    assert not res.converged and res.iterations == 2
    r = np.linalg.norm(g - A @ x.cpu().numpy()) / np.linalg.norm(g)
    assert abs(r - res.rel_residual) <= 1e-6 * r
    _, res = ws.solve(cu(nz), cu(g), tol=1e-8, maxit=0)
    assert not res.converged and res.iterations == 0 and abs(res.rel_residual - 1.0) <= 1e-14
    x, res = ws.solve(cu(nz), torch.zeros(st.nr, dtype=torch.float64, device="cuda"), cu(g))
    assert res.converged and res.iterations == 0 and not x.any()
    bad = nz.copy()
    for block in (31, 17):
        bad[pat.diag_inds[6 * block + 4]] = -1.0
    x0 = cu(g.copy())
    x, res = ws.solve(cu(bad), cu(g), x0)
    assert not res.converged and res.failed_block == 18 and torch.equal(x, cu(g))
