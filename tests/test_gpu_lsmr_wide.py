"""LSMR's pass over J~ where its split changes: tables of few and of many couplings, so that one, two, four or eight lanes
share a row or a column, for each size of chunk and for tables larger than any, F on and off a 16-byte boundary's staging.
Solutions as in test_gpu_lsmr.py (1e-6 in the norm against the direct solution).

An iteration reads J~ once for both of its products. It may not take longer than the two products do as calls of their
own (each reads J~); the factor of 1.3 is room for the iteration's vector updates and its host read."""
import numpy as np
import pytest
import torch

from test_gpu_lsmr import close, direct
from test_gpu_qr import cu
from test_gpu_qr_paths import _fx, fill_tables

pytestmark = pytest.mark.gpu

SIZES = {   # couplings of the tables, cameras; 6 variables a camera unless said
    "one table of one camera": (1, [1], 6),
    "chunks of 64 KB": (45, [1 + i % 9 for i in range(40)], 6),
    "one in chunks of 104 KB": (45, [27, 29, 28, 3, 30, 1, 31, 12], 6),
    "chunks of 208 KB": (45, [33, 38, 40, 2, 36, 41], 6),
    "3-variable cameras": (90, [55, 56, 5, 54, 1, 2, 57], 3),
}


def problem(bls, name, seed=7):
    cams, sizes, d = SIZES[name]
    rng = np.random.default_rng(seed)
    fx = _fx(rng, [d] * cams, [3] * len(sizes), sizes)
    st = bls.SchurStructure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    return bls.SchurJacobianStructure.positional(st, fx["e_rows"]), rng


@pytest.mark.parametrize("bulk", [True, False], ids=["bulk", "elements"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", list(SIZES))
def test_vs_direct(bls, name, dtype, bulk):
    j, rng = problem(bls, name)
    Rw, Rr, _, _ = fill_tables(j, rng)
    ws = bls.QRReductionWorkspace(j, None, dtype)
    ws.set_staging(bulk)
    s_r = 0.5 + rng.random(j.schur.nr)
    assert bls.reduce_qr(ws, bls.SchurBlockJacobian(j, dtype, data=cu(Rw, dtype), r=cu(Rr)), cu(0.5 + rng.random(j.schur.ne)), 1e-2)
    ref, _ = direct(bls, ws, 1e-2, s_r)
    x = torch.full((j.schur.nr,), float("nan"), dtype=torch.float64, device="cuda")
    for _ in range(2):
        res = bls.lsmr_reduced(x, ws, 1e-2, cu(s_r), atol=1e-12, btol=1e-12, conlim=1e14)
        assert res.solved and close(x.cpu().numpy(), ref, 1e-6), res


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("kmin,kmax,tables", [(4, 8, 20000), (18, 30, 3000), (25, 34, 2500)])
def test_an_iteration_against_its_products(bls, kmin, kmax, tables, dtype):
    rng = np.random.default_rng(kmin)
    cams = 120
    sizes = rng.integers(kmin, kmax + 1, tables)
    order = np.argsort(rng.random((tables, cams)), axis=1)
    coup = [sorted(order[i, :k].tolist()) for i, k in enumerate(sizes)]
    st = bls.SchurStructure.positional([6] * cams, [3] * tables, coup)
    j = bls.SchurJacobianStructure.positional(st, (2 * sizes).tolist())
    ws = bls.QRReductionWorkspace(j, None, dtype)
    gen = torch.Generator(device="cuda").manual_seed(1)
    data = torch.randn(j.raw_length, dtype=dtype, device="cuda", generator=gen)
    r = torch.randn(j.residual_length, dtype=torch.float64, device="cuda", generator=gen)
    assert bls.reduce_qr(ws, bls.SchurBlockJacobian(j, dtype, data=data, r=r), torch.ones(st.ne, dtype=torch.float64, device="cuda"), 1e-2)
    x = torch.zeros(st.nr, dtype=torch.float64, device="cuda")
    y = torch.zeros(bls.reduced_nrows(j), dtype=torch.float64, device="cuda")

    def median(f):
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            f()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return float(np.median(times[2:]))

    solve = lambda n: bls.lsmr_reduced(x, ws, 1e-6, None, atol=0.0, btol=0.0, conlim=1e300, itmax=n)
    assert solve(12).iterations == 12
    iteration = (median(lambda: solve(12)) - median(lambda: solve(2))) / 10
    products = median(lambda: bls.reduced_mul(y, ws, x)) + median(lambda: bls.reduced_tmul(x, ws, y))
    assert iteration <= 1.3 * products, (iteration, products)
