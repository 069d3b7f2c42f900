"""FP32 columns of S that the runs split over several items: S holds R, and each item's part is small beside it, so the
diagonal block is subtracted once. Points that see few of few cameras make columns of many visits.

Error of a diagonal block against 64 bits: R - c with c = C' E^-1 C summed in FP32 and R stored exactly. One subtraction
rounds c and the difference, 2 u of R at most with c <= R (u = 2^-24); the sum of c over n visits, by threads, warps and
items, adds a few u of c. In the norm over many entries roundings average to 1/sqrt(3) of their bound and better; 1.5 u is
asked for. A subtraction per item rounds S once more for each of them."""
import numpy as np
import pytest
import torch

import oracle as orc
from fixtures import make_problem, split_hessian
from test_gpu_column_runs import couplings
from test_gpu_schur import cu, relerr

pytestmark = pytest.mark.gpu


def tall(bls, nr, ne, r_dim, e_dim, dense, seed):
    """(S, g, oracle S, oracle g, diagonal-block entries) in the mixed form. H is a sum over visits (its diagonal blocks
    grow with them), not the dominant fixture: C of unit size, E a few times C'C, R above C' E^-1 C."""
    rng = np.random.default_rng(seed)
    r_dims, e_dims, coup = [r_dim] * nr, [e_dim] * ne, couplings(rng, nr, ne, 2, 4)
    st = bls.SchurStructure.positional(r_dims, e_dims, coup)
    ost = orc.Structure.positional(r_dims, e_dims, coup)
    pat, opat = bls.build_schur_pattern(st), orc.Pattern(ost)
    f4 = lambda a: a.astype(np.float32).astype(np.float64)
    E = np.zeros(st.E_length)
    C = np.zeros(st.C_length)
    blocks = np.zeros((nr, r_dim, r_dim))
    for e in range(ne):
        Jp = rng.standard_normal((len(coup[e]), 2, e_dim))
        Jc = rng.standard_normal((len(coup[e]), 2, r_dim))
        E[e * e_dim**2:(e + 1) * e_dim**2] = (np.einsum("kia,kib->ab", Jp, Jp) + np.eye(e_dim)).ravel()
        for k, r in enumerate(coup[e]):
            c = int(st.eliminated_ptr[e]) + k
            C[c * r_dim * e_dim:(c + 1) * r_dim * e_dim] = (Jp[k].T @ Jc[k]).ravel(order="F")
            blocks[r] += Jc[k].T @ Jc[k]
    E, C, blocks = f4(E), f4(C), f4(blocks)
    n = st.nr
    if dense:
        R = np.zeros((n, n))
        for r in range(nr):
            R[r * r_dim:(r + 1) * r_dim, r * r_dim:(r + 1) * r_dim] = blocks[r]
        R = R.ravel(order="F")
    else:
        R = np.zeros(pat.R_length)
        for r in range(nr):
            s = int(pat.R_block_start[pat.block_colptr[r + 1] - 1])
            R[s:s + r_dim**2] = blocks[r].ravel(order="F")
    b_r, b_e = rng.standard_normal(n), rng.standard_normal(st.ne)
    sc_r, sc_e, lam = np.zeros(n), np.zeros(st.ne), 0.0
    ws = bls.SchurReductionWorkspace(st, None if dense else pat)
    t = lambda a: cu(a.astype(np.float32))
    S = torch.zeros(n * n if dense else pat.nnz, dtype=torch.float32, device="cuda")
    g = torch.zeros(n, dtype=torch.float64, device="cuda")
    oS, og, work = np.zeros(S.numel()), np.zeros(n), orc.Work(ost, 1)
    for _ in range(2):   # the second call starts from what the first one left in the plan
        if dense:
            bls.reset_schur_dense(S, t(R), cu(sc_r), lam, ws)
            assert bls.reduce_schur_dense(S, g, cu(b_r), cu(b_e), cu(sc_e), lam, st, t(E), t(C), ws)
        else:
            bls.reset_schur_sparse(S, t(R), None, None, cu(sc_r), lam, ws)
            assert bls.reduce_schur_sparse(S, g, cu(b_r), cu(b_e), cu(sc_e), lam, st, t(E), t(C), None, None, None, None, ws)
    if dense:
        orc.reset_schur_dense(ost, oS, R, sc_r, lam, None)
        ok, _ = orc.reduce_schur_dense(ost, work, oS, og, b_r, b_e, sc_e, lam, E, C, None, None)
        rows, cols = np.tile(np.arange(n), n), np.repeat(np.arange(n), n)
    else:
        orc.reset_schur_sparse(ost, opat, oS, R, sc_r, lam, None)
        ok, _ = orc.reduce_schur_sparse(ost, opat, work, oS, og, b_r, b_e, sc_e, lam, E, C, None, None)
        rows, cols = pat.S_rowval, np.repeat(np.arange(n), np.diff(pat.S_colptr))
    assert ok
    diag = (rows // r_dim == cols // r_dim) & (rows <= cols)
    return S.double().cpu().numpy(), g.cpu().numpy(), oS, og, diag, ws.phase2_kernel_name(torch.float32, dense=dense)


@pytest.mark.parametrize("dense", [False, True], ids=["sparse", "dense"])
@pytest.mark.parametrize("r_dim,e_dim", [(6, 3), (9, 3), (5, 2)])
def test_diagonal_blocks_of_split_columns(bls, r_dim, e_dim, dense):
    S, g, oS, og, diag, kernel = tall(bls, 8, 6000, r_dim, e_dim, dense, 3)
    assert kernel.startswith("k_runs")
    assert relerr(g, og) <= 1e-10
    assert np.linalg.norm((S - oS)[diag]) <= 1.5 * 2.0**-24 * np.linalg.norm(oS[diag])
    assert relerr(S, oS) <= 1e-4
