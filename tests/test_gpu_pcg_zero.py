"""PCG with g = 0 from a non-zero start: the solution is x = 0 and no iteration is spent on it (none reaches a residual of
exactly zero). Its time is held against a solve that may not iterate: the starts are the same, the factor of 4 is room for
the host."""
import numpy as np
import pytest
import torch

from test_gpu_pcg_columns import system
from test_gpu_schur import cu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncam,npts,kmax", [(7, 40, 4), (190, 900, 30), (401, 3000, 5)])
def test_no_iterations_for_a_zero_right_hand_side(bls, ncam, npts, kmax):
    st, pat, nz, _ = system(bls, ncam, npts, kmax, 9)
    rng = np.random.default_rng(3)
    ws, S, g, x0 = bls.PCGWorkspace(st, pat), cu(nz), cu(rng.standard_normal(st.nr)), cu(rng.standard_normal(st.nr))

    def median(g, maxit):
        times = []
        for _ in range(15):
            x = x0.clone()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            x, res = ws.solve(S, g, x, tol=1e-8, maxit=maxit)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return float(np.median(times)), x, res

    start, _, _ = median(g, 0)
    zero, x, res = median(torch.zeros_like(g), 1000)
    assert res.converged and res.iterations == 0 and res.rel_residual == 0.0 and not x.any()
    assert zero <= 4 * start
