"""Plans keep their small device arrays in one allocation: plans of several sizes (all arrays small, some large) alive at the
same time and released in another order than they were made, schedules added by choosing a kernel by name, repeatedly, and
the reductions of the remaining plans unchanged by any of it (bit for bit where a column has one item, 1e-12 of the largest
entry otherwise: additions of split columns are unordered)."""
import gc

import numpy as np
import pytest
import torch

from fixtures import make_problem, split_hessian
from test_gpu_column_runs import couplings
from test_gpu_schur import cu, relerr

pytestmark = pytest.mark.gpu


class Problem:
    def __init__(self, bls, r_dim, nr, ne, kmin, kmax, dense):
        rng = np.random.default_rng(nr + ne)
        self.bls, self.dense = bls, dense
        r_dims, e_dims, coup = [r_dim] * nr, [3] * ne, couplings(rng, nr, ne, kmin, kmax)
        H, b = make_problem(rng, r_dims, e_dims, coup)
        self.st = st = bls.SchurStructure.positional(r_dims, e_dims, coup)
        pat = None if dense else bls.build_schur_pattern(st)
        self.E, self.C, self.R = (cu(a) for a in split_hessian(H, st, pat))
        n = st.nr
        self.sc_r, self.sc_e, self.b_r, self.b_e = cu(np.diag(H)[:n].copy()), cu(np.diag(H)[n:].copy()), cu(b[:n]), cu(b[n:])
        self.ws = bls.SchurReductionWorkspace(st, pat)
        self.S = torch.zeros(n * n if dense else pat.nnz, dtype=torch.float64, device="cuda")
        self.g = torch.zeros(n, dtype=torch.float64, device="cuda")

    def reduce(self):
        b, a = self.bls, (self.g, self.b_r, self.b_e, self.sc_e, 1e-3, self.st, self.E, self.C)
        if self.dense:
            b.reset_schur_dense(self.S, self.R, self.sc_r, 1e-3, self.ws)
            assert b.reduce_schur_dense(self.S, *a, self.ws)
        else:
            b.reset_schur_sparse(self.S, self.R, None, None, self.sc_r, 1e-3, self.ws)
            assert b.reduce_schur_sparse(self.S, *a, None, None, None, None, self.ws)
        return self.S.cpu().numpy(), self.g.cpu().numpy()


def test_plans_side_by_side(bls):
    shapes = [(6, 5, 40, 1, 4, False), (9, 40, 900, 2, 9, False), (6, 60, 1500, 2, 12, True), (6, 120, 1200, 2, 20, False), (7, 3, 9, 1, 3, False),
              (6, 80, 1400, 8, 16, False)]
    problems = [Problem(bls, *s) for s in shapes]
    want = [p.reduce() for p in problems]
    for p, s in zip(problems, shapes):
        if s[0] == 6 and not s[5]:
            for kernel in ("runs", "gather", "runs", "pairs", "gather", "stage"):
                p.ws.set_kernel(kernel)
                S, g = p.reduce()
                w = want[problems.index(p)]
                assert relerr(S, w[0]) <= 1e-12 and relerr(g, w[1]) <= 1e-12, kernel
    for i in (3, 0, 5, 1):   # release some, make another one, use the rest
        problems[i] = None
        gc.collect()
        extra = Problem(bls, 6, 30 + i, 300, 1, 8, False)
        extra.reduce()
        for p, w in zip(problems, want):
            if p is not None:
                S, g = p.reduce()
                assert relerr(S, w[0]) <= 1e-12 and relerr(g, w[1]) <= 1e-12
