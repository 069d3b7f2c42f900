"""qr_backsubstitute where its lanes are dealt differently: retained blocks of 1, 2, 3 to 4 and more variables, eliminated
ones of 1, up to 4, up to 8 and more, against the oracle on the same stored tables (tolerances as in test_gpu_qr.py).

1-variable cameras with the same couplings are a sixth of the data of 6-variable ones; finding the entries is the same work.
They may take half the time at most."""
import numpy as np
import pytest
import torch

import oracle as orc
from test_gpu_qr import check_close, run_both
from test_gpu_qr_paths import _fx, fill_tables

pytestmark = pytest.mark.gpu

SIZES = {"1x1": ([1], [1]), "1x3": ([1], [3]), "2x5": ([2], [5]), "3x8": ([3], [8]), "4x9": ([4], [9]), "5x1": ([5], [1]), "1 to 16 by 17 to 1": (list(range(1, 17)), [17, 8, 4, 1])}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
@pytest.mark.parametrize("name", list(SIZES))
def test_vs_oracle(bls, name, dtype):
    rng = np.random.default_rng(37)
    r, e = SIZES[name]
    r_dims, e_dims = (r * 16)[:16], sorted((e * 40)[:40], reverse=True)
    fx = _fx(rng, r_dims, e_dims, [1 + i % 9 for i in range(40)])
    st = bls.SchurStructure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    ost = orc.Structure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    j, o = bls.SchurJacobianStructure.positional(st, fx["e_rows"]), orc.QRStructure.positional(ost, fx["e_rows"])
    Rw, Rr, _, _ = fill_tables(j, rng)
    check_close(run_both(bls, j, o, Rw, Rr, 0.5 + rng.random(j.schur.ne), 1e-3, dtype), 1e-12 if dtype == torch.float64 else 1e-5)


def test_small_blocks_against_larger_ones(bls):
    rng = np.random.default_rng(2)
    cams, points = 300, 60000
    k = rng.integers(2, 9, points)
    first = rng.integers(0, cams - 40, points)
    coup = [sorted((first[i] + rng.permutation(40)[:k[i]]).tolist()) for i in range(points)]
    times = {}
    for d in (1, 6):
        st = bls.SchurStructure.positional([d] * cams, [3] * points, coup)
        j = bls.SchurJacobianStructure.positional(st, (2 * k).tolist())
        ws = bls.QRReductionWorkspace(j, None, torch.float64)
        f8 = dict(dtype=torch.float64, device="cuda")
        assert bls.reduce_qr(ws, bls.SchurBlockJacobian(j, torch.float64, data=torch.randn(j.raw_length, **f8), r=torch.randn(j.residual_length, **f8)), torch.ones(st.ne, **f8), 1e-2)
        x_r, x_e, t = torch.randn(st.nr, **f8), torch.zeros(st.ne, **f8), []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            bls.qr_backsubstitute(x_e, x_r, ws)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        times[d] = float(np.median(t[3:]))
    assert times[1] <= 0.5 * times[6], times
