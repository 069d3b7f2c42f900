"""J~'J~ and its diagonal blocks for retained sizes other than 6, where the products' split in blocks of eight rows and three
columns ends (1 to 4, 7, 8, 9, 15, 16 and mixtures), against the oracle on the same stored tables. Tolerances as in
test_gpu_qr.py (1e-12 relative in FP64, 1e-5 in the mixed form).

The mixed form reads half the bytes of FP64 and adds a conversion per entry to the same FP64 products: its diagonal blocks
may not take more than twice as long."""
import numpy as np
import pytest
import torch

from test_gpu_qr import check_close, run_both
from test_gpu_qr_paths import _fx, fill_tables
import oracle as orc

pytestmark = pytest.mark.gpu

DIMS = {"1": [1], "2 and 3": [2, 3], "4": [4], "7": [7], "8": [8], "9": [9], "9 and 6": [9, 6], "15 and 16": [15, 16], "1 to 16": list(range(1, 17))}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", list(DIMS))
def test_vs_oracle(bls, name, dtype):
    rng = np.random.default_rng(29)
    r_dims = (DIMS[name] * 16)[:16]
    fx = _fx(rng, r_dims, [3] * 45, [1 + i % 7 for i in range(45)])
    st = bls.SchurStructure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    ost = orc.Structure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    j = bls.SchurJacobianStructure.positional(st, fx["e_rows"])
    o = orc.QRStructure.positional(ost, fx["e_rows"])
    Rw, Rr, _, _ = fill_tables(j, rng)
    check_close(run_both(bls, j, o, Rw, Rr, 0.5 + rng.random(j.schur.ne), 1e-3, dtype), 1e-12 if dtype == torch.float64 else 1e-5)


@pytest.mark.parametrize("d", [3, 7, 9])
def test_diagonal_blocks_of_both_forms(bls, d):
    rng = np.random.default_rng(d)
    cams, tables = 100, 12000
    sizes = rng.integers(3, 9, tables)
    order = np.argsort(rng.random((tables, cams)), axis=1)
    st = bls.SchurStructure.positional([d] * cams, [3] * tables, [sorted(order[i, :k].tolist()) for i, k in enumerate(sizes)])
    j = bls.SchurJacobianStructure.positional(st, (2 * sizes).tolist())
    times = {}
    for dtype in (torch.float64, torch.float32):
        ws = bls.QRReductionWorkspace(j, None, dtype)
        gen = torch.Generator(device="cuda").manual_seed(1)
        data = torch.randn(j.raw_length, dtype=dtype, device="cuda", generator=gen)
        r = torch.randn(j.residual_length, dtype=torch.float64, device="cuda", generator=gen)
        assert bls.reduce_qr(ws, bls.SchurBlockJacobian(j, dtype, data=data, r=r), torch.ones(st.ne, dtype=torch.float64, device="cuda"), 1e-2)
        D = torch.zeros(int(j.doffsets[-1]), dtype=dtype, device="cuda")
        t = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            bls.reduced_diagonal_blocks(D, ws)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        times[dtype] = float(np.median(t[2:]))
    assert times[torch.float32] <= 2 * times[torch.float64], times
