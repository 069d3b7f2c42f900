"""Two host threads, each with plans of its own, reducing at the same time: a kernel's shared-memory limit belongs to the
process, so a launch of the smaller plan must not lower it under the larger plan's launch. What each thread computes is
compared with the same calls made alone (additions of split columns are unordered: 1e-12 of the largest entry in FP64)."""
import threading
import time

import numpy as np
import pytest
import torch

from fixtures import make_problem, split_hessian
from test_gpu_column_runs import couplings
from test_gpu_schur import cu, relerr

pytestmark = pytest.mark.gpu


def caller(bls, r_dim, nr, ne, kmin, kmax, kernel):
    """A function of no arguments that resets and reduces into buffers of its own and returns (S, g)."""
    rng = np.random.default_rng(nr)
    fx = dict(r_dims=[r_dim] * nr, e_dims=[3] * ne, couplings=couplings(rng, nr, ne, kmin, kmax))
    H, b = make_problem(rng, fx["r_dims"], fx["e_dims"], fx["couplings"])
    st = bls.SchurStructure.positional(fx["r_dims"], fx["e_dims"], fx["couplings"])
    pat = bls.build_schur_pattern(st)
    E, Cd, R = (cu(a) for a in split_hessian(H, st, pat))
    sc_r, sc_e, b_r, b_e = cu(np.diag(H)[:st.nr].copy()), cu(np.diag(H)[st.nr:].copy()), cu(b[:st.nr]), cu(b[st.nr:])
    ws = bls.SchurReductionWorkspace(st, pat)
    ws.set_kernel(kernel)
    S = torch.zeros(pat.nnz, dtype=torch.float64, device="cuda")
    g = torch.zeros(st.nr, dtype=torch.float64, device="cuda")

    def call(times=1):
        for _ in range(times):
            bls.reset_schur_sparse(S, R, None, None, sc_r, 1e-3, ws)
            bls.reduce_schur_sparse(S, g, b_r, b_e, sc_e, 1e-3, st, E, Cd, None, None, None, None, ws, sync=False)
        assert ws.query_status()
        return S.cpu().numpy(), g.cpu().numpy()

    return call


@pytest.mark.parametrize("r_dim,nr,k,kernel", [(9, 120, 80, "stage"), (6, 260, 125, "runs"), (6, 260, 125, "gather")])
def test_plans_of_two_sizes(bls, r_dim, nr, k, kernel):
    # the second plan's columns are tall: its launches take more shared memory than the first one's
    calls = [caller(bls, r_dim, 4, 30, 1, 3, kernel), caller(bls, r_dim, nr, 14, k - 3, k, kernel)]
    want = [c() for c in calls]
    got, errors, end = [None, None], [], time.monotonic() + 5

    def work(i):
        try:
            while time.monotonic() < end and not errors:   # the moment between setting the limit and the launch is short
                got[i] = calls[i](100)
        except Exception as e:   # reported by the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for (S, g), (S0, g0) in zip(got, want):
        assert relerr(S, S0) <= 1e-12 and relerr(g, g0) <= 1e-12
