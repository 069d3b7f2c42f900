"""The QR route's kernels where their split changes, against the oracle on the same stored tables: J~'J~ of tables with
at most and with more than 16 pairs of 6 x 6 blocks in one size class (a lane per block column or per whole block, FP32
additions of two and four values), one and many cameras per table, sizes other than 6; the back-substitution's eight lanes
and its rows by 4 and 16 (eliminated sizes 1, 4, 5, 16, 17 and 33); LSMR's chunks of tables (a table larger than a chunk,
chunks of many small ones, element reads instead of bulk copies).

Tolerances as in test_gpu_qr.py (1e-12 relative in FP64, 1e-5 in the mixed form) and, for LSMR, as in test_gpu_lsmr.py
(1e-6 in the norm against the direct solution)."""
import numpy as np
import pytest
import torch

import oracle as orc
from qr_fixtures import fill_tables
from test_gpu_lsmr import close, direct
from test_gpu_qr import check_close, cu, run_both

pytestmark = pytest.mark.gpu


def _coup(rng, nr, sizes):
    return [sorted(rng.choice(nr, size=k, replace=False).tolist()) for k in sizes]


def _fx(rng, r_dims, e_dims, sizes, extra=3, **kw):
    c = _coup(rng, len(r_dims), sizes)
    rows = [max(2 * len(x), d + extra) for x, d in zip(c, e_dims)]
    return dict(r_dims=r_dims, e_dims=e_dims, couplings=c, e_rows=rows, **kw)


def structures():
    rng = np.random.default_rng(23)
    return {
        "6x3, 1 to 12 cameras": _fx(rng, [6] * 14, [3] * 90, [1 + i % 12 for i in range(90)]),
        "6x3, 5 and 6 cameras": _fx(rng, [6] * 9, [3] * 64, [5 + i % 2 for i in range(64)]),
        "6x3, 31 to 33 cameras": _fx(rng, [6] * 40, [3] * 21, [31 + i % 3 for i in range(21)]),
        "9 and 6 by 1 to 4": _fx(rng, [9, 6] * 5, [1 + i % 4 for i in range(45)], [1 + i % 7 for i in range(45)]),
        "eliminated to 33": _fx(rng, [6] * 6, [4, 5, 16, 17, 33, 1, 20, 32], [1, 2, 3, 2, 3, 1, 6, 2]),
        "free groups": _fx(rng, [6] * 10, [3] * 40, [2 + i % 5 for i in range(40)], free_rows=[9, 80, 4],
                           free_retained=[[1, 0], [4, 5, 6, 7, 8, 9], [3]]),
    }


STRUCTURES = structures()


def build(bls, name):
    fx = STRUCTURES[name]
    rng = np.random.default_rng(3)
    st = bls.SchurStructure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    ost = orc.Structure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    free = (fx.get("free_rows", ()), fx.get("free_retained", ()))
    j = bls.SchurJacobianStructure.positional(st, fx["e_rows"], *free)
    o = orc.QRStructure.positional(ost, fx["e_rows"], *free)
    Rw, Rr, _, _ = fill_tables(j, rng)
    return j, o, Rw, Rr, 0.5 + rng.random(j.schur.ne), 0.5 + rng.random(j.schur.nr)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", list(STRUCTURES))
def test_gram_and_backsubstitution_vs_oracle(bls, name, dtype):
    j, o, Rw, Rr, sc_e, _ = build(bls, name)
    check_close(run_both(bls, j, o, Rw, Rr, sc_e, 1e-3, dtype), 1e-12 if dtype == torch.float64 else 1e-5)


@pytest.mark.parametrize("bulk", [True, False], ids=["bulk", "elements"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", list(STRUCTURES))
def test_lsmr_vs_direct(bls, name, dtype, bulk):
    j, _, Rw, Rr, sc_e, s_r = build(bls, name)
    ws = bls.QRReductionWorkspace(j, None, dtype)
    ws.set_staging(bulk)
    J = bls.SchurBlockJacobian(j, dtype, data=cu(Rw, dtype), r=cu(Rr))
    for lam in (1e-3, 1.0):
        assert bls.reduce_qr(ws, J, cu(sc_e), lam)
        ref, _ = direct(bls, ws, lam, s_r)
        x = torch.full((j.schur.nr,), float("nan"), dtype=torch.float64, device="cuda")
        res = bls.lsmr_reduced(x, ws, lam, cu(s_r), atol=1e-12, btol=1e-12, conlim=1e14)
        assert res.solved and close(x.cpu().numpy(), ref, 1e-6), (lam, res)
        # a second solve on the same workspace, undisturbed by what the first left in it
        y = torch.full_like(x, float("nan"))
        assert bls.lsmr_reduced(y, ws, lam, cu(s_r), atol=1e-12, btol=1e-12, conlim=1e14).solved
        assert close(y.cpu().numpy(), ref, 1e-6)
