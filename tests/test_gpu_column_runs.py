"""Phase 2 of the Schur reduction with the couplings of a column's points staged in shared memory ("runs"), against the
oracle on the same stored values, where its schedule and its copies can go wrong: every exact block size (6 to 9 with 3)
and mixed sizes up to 16, a single camera, points that see one camera or nearly all of them (several segments per item,
several lanes per block), couplings whose storage ends inside a 16-byte chunk, C off a 16-byte boundary (the kernel is
not used there), both storage types, sparse and dense S, conditioning scales.

Tolerances as in test_gpu_schur.py: 1e-12 relative in FP64; in the mixed form 1e-4 in S (FP32 accumulation of ~k^2 terms
of size |C|^2 / |E|) and 1e-10 in g_S, which is formed in FP64 from the FP32-rounded inputs on both sides."""
import numpy as np
import pytest
import torch

import oracle as orc
from fixtures import make_problem, split_hessian
from test_gpu_schur import cu, relerr

pytestmark = pytest.mark.gpu


def couplings(rng, nr, ne, kmin, kmax):
    return [sorted(rng.choice(nr, size=min(nr, int(rng.integers(kmin, kmax + 1))), replace=False).tolist()) for _ in range(ne)]


def structures():
    rng = np.random.default_rng(5)
    out = {f"uniform {d}x3": dict(r_dims=[d] * 21, e_dims=[3] * 83, couplings=couplings(rng, 21, 83, 1, 7)) for d in (6, 7, 8, 9)}
    out["one camera"] = dict(r_dims=[9], e_dims=[3] * 37, couplings=[[0]] * 37)
    out["long runs 6x3"] = dict(r_dims=[6] * 64, e_dims=[3] * 40, couplings=couplings(rng, 64, 40, 40, 60))
    out["long runs 9x3"] = dict(r_dims=[9] * 30, e_dims=[3] * 41, couplings=couplings(rng, 30, 41, 20, 29))
    out["two cameras"] = dict(r_dims=[6] * 2, e_dims=[3] * 301, couplings=couplings(rng, 2, 301, 1, 2))
    out["mixed 9,6 by 3,1"] = dict(r_dims=[9, 6] * 8, e_dims=[3] * 50 + [1] * 49, couplings=couplings(rng, 16, 99, 1, 6))
    out["mixed to 16"] = dict(r_dims=[16, 1, 11, 6, 3], e_dims=[16, 12, 9, 8, 5, 4, 3, 2, 1, 1, 1], couplings=couplings(rng, 5, 11, 1, 4))
    out["uniform 16x3"] = dict(r_dims=[16] * 7, e_dims=[3] * 60, couplings=couplings(rng, 7, 60, 1, 5))
    return out


STRUCTURES = structures()


def reduce_both(bls, fx, dtype, dense, scaled, kernel, offset=0, unit=None):
    """(S, g, oracle S, oracle g, name of the kernel) of one reset + reduce; `offset` entries in front of C."""
    rng = np.random.default_rng(17)
    npdt = np.float32 if dtype == torch.float32 else np.float64
    H, b = make_problem(rng, fx["r_dims"], fx["e_dims"], fx["couplings"])
    st = bls.SchurStructure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    ost = orc.Structure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    pat, opat = bls.build_schur_pattern(st), orc.Pattern(ost)
    E, Cd, R = (a.astype(npdt) for a in split_hessian(H, st, None if dense else pat))
    nr, ne, lam = st.nr, st.ne, 1e-3
    sc_r, sc_e = np.diag(H)[:nr].copy(), np.diag(H)[nr:].copy()
    s_r = 2.0 ** rng.integers(-3, 4, nr) if scaled else None
    s_e = 2.0 ** rng.integers(-3, 4, ne) if scaled else None
    dv = lambda a: None if a is None else cu(a)
    ws = bls.SchurReductionWorkspace(st, pat)
    ws.set_kernel(kernel)
    if unit is not None:
        ws.set_stage_unit(unit)
    buf = torch.zeros(offset + Cd.size, dtype=dtype, device="cuda")
    buf[offset:] = cu(Cd)
    g = torch.zeros(nr, dtype=torch.float64, device="cuda")
    S = torch.zeros(nr * nr if dense else pat.nnz, dtype=dtype, device="cuda")
    args = (g, cu(b[:nr]), cu(b[nr:]), cu(sc_e), lam, st, cu(E), buf[offset:])
    if dense:
        bls.reset_schur_dense(S, cu(R), cu(sc_r), lam, ws, s_r=dv(s_r))
        assert bls.reduce_schur_dense(S, *args, ws, s_r=dv(s_r), s_e=dv(s_e))
    else:
        bls.reset_schur_sparse(S, cu(R), None, None, cu(sc_r), lam, ws, s_r=dv(s_r))
        assert bls.reduce_schur_sparse(S, *args, None, None, None, None, ws, s_r=dv(s_r), s_e=dv(s_e))
    f8 = lambda a: a.astype(np.float64)
    oS, og, work = np.zeros(S.numel()), np.zeros(nr), orc.Work(ost, 1)
    if dense:
        orc.reset_schur_dense(ost, oS, f8(R), sc_r, lam, s_r)
        ok, _ = orc.reduce_schur_dense(ost, work, oS, og, b[:nr], b[nr:], sc_e, lam, f8(E), f8(Cd), s_r, s_e)
    else:
        orc.reset_schur_sparse(ost, opat, oS, f8(R), sc_r, lam, s_r)
        ok, _ = orc.reduce_schur_sparse(ost, opat, work, oS, og, b[:nr], b[nr:], sc_e, lam, f8(E), f8(Cd), s_r, s_e)
    assert ok
    return S.double().cpu().numpy(), g.cpu().numpy(), oS, og, ws.phase2_kernel_name(dtype, dense=dense)


@pytest.mark.parametrize("scaled", [False, True], ids=["plain", "scaled"])
@pytest.mark.parametrize("dense", [False, True], ids=["sparse", "dense"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", list(STRUCTURES))
def test_runs_against_oracle(bls, name, dtype, dense, scaled):
    S, g, oS, og, kernel = reduce_both(bls, STRUCTURES[name], dtype, dense, scaled, "runs")
    assert kernel.startswith("k_runs")
    f64 = dtype == torch.float64
    assert relerr(S, oS) <= (1e-12 if f64 else 1e-4)
    assert relerr(g, og) <= (1e-12 if f64 else 1e-10)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", ["uniform 6x3", "uniform 9x3", "mixed 9,6 by 3,1"])
def test_unaligned_couplings(bls, name, dtype):
    """C two elements past a 16-byte boundary (FP64: one past it, where the plan's sizes take single elements) is still
    accepted and reduced, by another kernel."""
    offset = 2 if dtype == torch.float32 else 1
    fx = STRUCTURES[name]
    if name == "uniform 6x3" and dtype == torch.float64:
        pytest.skip("6 x 3 blocks in FP64 need C on two elements, a 16-byte boundary")
    S, g, oS, og, _ = reduce_both(bls, fx, dtype, False, False, "stage", offset)
    assert relerr(S, oS) <= (1e-12 if dtype == torch.float64 else 1e-4)
    assert relerr(g, og) <= (1e-12 if dtype == torch.float64 else 1e-10)


@pytest.mark.parametrize("unit", [None, 1, 24])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
def test_gather_form(bls, dtype, unit):
    """The other column-owned kernel, which "stage" takes by the plan's sizes, named directly (its schedule is then
    built from the plan's device copies)."""
    S, g, oS, og, kernel = reduce_both(bls, STRUCTURES["uniform 6x3"], dtype, False, True, "gather", unit=unit)
    assert kernel.startswith("k_stage36")
    assert relerr(S, oS) <= (1e-12 if dtype == torch.float64 else 1e-4)
    assert relerr(g, og) <= (1e-12 if dtype == torch.float64 else 1e-10)


@pytest.mark.parametrize("scaled", [False, True], ids=["plain", "scaled"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", list(STRUCTURES))
def test_backsubstitution(bls, name, dtype, scaled):
    """x_e of every structure against its definition in FP64 numpy from the same stored values (z - E^-1 C x_r, with the
    scaled blocks rounded to the storage type; power-of-two scales, so the rounding is exact): 1e-12 relative, FP64 sums
    of at most 60 x 9 products behind an inverse of condition below 10."""
    fx = STRUCTURES[name]
    rng = np.random.default_rng(23)
    npdt = np.float32 if dtype == torch.float32 else np.float64
    H, b = make_problem(rng, fx["r_dims"], fx["e_dims"], fx["couplings"])
    st = bls.SchurStructure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    pat = bls.build_schur_pattern(st)
    E, Cd, R = (a.astype(npdt) for a in split_hessian(H, st, pat))
    nr, ne, lam = st.nr, st.ne, 1e-3
    sc = np.diag(H).copy()
    s = 2.0 ** rng.integers(-2, 3, nr + ne) if scaled else np.ones(nr + ne)
    dv = (lambda a: cu(a)) if scaled else (lambda a: None)
    ws = bls.SchurReductionWorkspace(st, pat)
    g, S = torch.zeros(nr, dtype=torch.float64, device="cuda"), torch.zeros(pat.nnz, dtype=dtype, device="cuda")
    bls.reset_schur_sparse(S, cu(R), None, None, cu(sc[:nr]), lam, ws, s_r=dv(s[:nr]))
    assert bls.reduce_schur_sparse(S, g, cu(b[:nr]), cu(b[nr:]), cu(sc[nr:]), lam, st, cu(E), cu(Cd), None, None, None, None, ws,
                                   s_r=dv(s[:nr]), s_e=dv(s[nr:]))
    x_r = rng.standard_normal(nr)
    x_e = torch.zeros(ne, dtype=torch.float64, device="cuda")
    bls.backsubstitute(x_e, cu(x_r), st, cu(Cd), ws, s_r=dv(s[:nr]), s_e=dv(s[nr:]))
    want = np.zeros(ne)
    for e in range(st.neblocks):
        de, so = int(st.e_dims[e]), int(st.boffsets_e[e])
        eo = int(st.eoffsets[e])
        v = np.arange(so, so + de)
        Ed = E[eo:eo + de * de].astype(np.float64).reshape(de, de).T * np.outer(s[nr + v], s[nr + v]) + np.diag(lam * sc[nr + v] * s[nr + v] ** 2)
        t = np.zeros(de)
        for c in range(int(st.eliminated_ptr[e]), int(st.eliminated_ptr[e + 1])):
            r = int(st.entry_retained[c])
            dr, ro, co = int(st.r_dims[r]), int(st.boffsets_r[r]), int(st.coffsets[c])
            t += (Cd[co:co + dr * de].astype(np.float64).reshape(dr, de) * np.outer(s[ro:ro + dr], s[nr + v])).T @ x_r[ro:ro + dr]
        want[v] = np.linalg.solve(Ed, b[nr + v] * s[nr + v] - t)
    assert relerr(x_e.cpu().numpy(), want) <= 1e-12
