"""Back-substitution of other block sizes than the exact ones: its eight lanes per point split over the couplings of a point
and the columns of a coupling by the largest retained block (1, 2, 3 to 4, 5 and more), eliminated blocks of 1, up to 4 and
up to 16, points without couplings among them, against the oracle. Tolerances as in test_gpu_schur.py.

With 1-variable blocks most of the work is finding the couplings. A point's couplings shared by eight lanes may not take
longer than one of six-variable cameras (six times the data) with the same couplings."""
import numpy as np
import pytest
import torch

import oracle as orc
from fixtures import make_problem, split_hessian
from test_gpu_column_runs import couplings
from test_gpu_schur import cu, relerr

pytestmark = pytest.mark.gpu

SIZES = {"1x1": ([1], [1]), "2x1": ([2], [1]), "2x2": ([2], [2]), "3x3": ([3], [3]), "4x3": ([4], [3]), "5x1": ([5], [1]), "5x4": ([5], [4]),
         "2x5": ([2], [5]), "1 to 4 by 3 and 1": ([1, 2, 3, 4], [3, 1]), "16 to 1 by 16 to 1": ([16, 9, 1], [16, 4, 1])}


@pytest.mark.parametrize("scaled", [False, True], ids=["plain", "scaled"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", list(SIZES))
def test_vs_oracle(bls, name, dtype, scaled):
    rng = np.random.default_rng(31)
    npdt = np.float32 if dtype == torch.float32 else np.float64
    r, e = SIZES[name]
    r_dims, e_dims = (r * 19)[:19], sorted((e * 41)[:41], reverse=True)
    coup = couplings(rng, 19, 41, 1, 18)
    H, b = make_problem(rng, r_dims, e_dims, coup)
    st = bls.SchurStructure.positional(r_dims, e_dims, coup)
    ost = orc.Structure.positional(r_dims, e_dims, coup)
    pat, opat = bls.build_schur_pattern(st), orc.Pattern(ost)
    E, C, R = (a.astype(npdt) for a in split_hessian(H, st, pat))
    nr, ne, lam = st.nr, st.ne, 1e-3
    sc_r, sc_e = np.diag(H)[:nr].copy(), np.diag(H)[nr:].copy()
    s_r = 2.0 ** rng.integers(-3, 4, nr) if scaled else None
    s_e = 2.0 ** rng.integers(-3, 4, ne) if scaled else None
    dv = lambda a: None if a is None else cu(a)
    ws = bls.SchurReductionWorkspace(st, pat)
    S, g = torch.zeros(pat.nnz, dtype=dtype, device="cuda"), torch.zeros(nr, dtype=torch.float64, device="cuda")
    bls.reset_schur_sparse(S, cu(R), None, None, cu(sc_r), lam, ws, s_r=dv(s_r))
    assert bls.reduce_schur_sparse(S, g, cu(b[:nr]), cu(b[nr:]), cu(sc_e), lam, st, cu(E), cu(C), None, None, None, None, ws, s_r=dv(s_r), s_e=dv(s_e))
    x_r = rng.standard_normal(nr)
    x_e = torch.full((ne,), float("nan"), dtype=torch.float64, device="cuda")
    bls.backsubstitute(x_e, cu(x_r), st, cu(C), ws, dv(s_r), dv(s_e))
    f8 = lambda a: a.astype(np.float64)
    oS, og, work, ox = np.zeros(opat.nnz), np.zeros(nr), orc.Work(ost, 1), np.zeros(ne)
    orc.reset_schur_sparse(ost, opat, oS, f8(R), sc_r, lam, s_r)
    ok, _ = orc.reduce_schur_sparse(ost, opat, work, oS, og, b[:nr], b[nr:], sc_e, lam, f8(E), f8(C), s_r, s_e)
    assert ok
    orc.backsubstitute(ost, work, ox, x_r, f8(C), s_r, s_e)
    assert relerr(x_e.cpu().numpy(), ox) <= (1e-12 if dtype == torch.float64 else 1e-6)


def test_small_blocks_against_larger_ones(bls):
    rng = np.random.default_rng(2)
    cams, points = 600, 150000
    k = rng.integers(2, 11, points)
    first = rng.integers(0, cams - 40, points)
    coup = [sorted((first[i] + rng.permutation(40)[:k[i]]).tolist()) for i in range(points)]
    times = {}
    for d in (1, 6):
        st = bls.SchurStructure.positional([d] * cams, [1] * points, coup)
        ws = bls.SchurReductionWorkspace(st, bls.build_schur_pattern(st))
        f8 = dict(dtype=torch.float64, device="cuda")
        C, x_r, x_e = torch.randn(st.C_length, **f8), torch.randn(st.nr, **f8), torch.zeros(st.ne, **f8)
        t = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            bls.backsubstitute(x_e, x_r, st, C, ws)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        times[d] = float(np.median(t[3:]))
    assert times[1] <= 0.75 * times[6], times
