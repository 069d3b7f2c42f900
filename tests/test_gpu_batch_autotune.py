"""The batch autotuner times every kernel that keeps per-problem failure, the gather at each unit size, and leaves the plan
on the one it reports; whatever it chooses, the batch's result is the same (tolerances as in test_gpu_batch.py)."""
import numpy as np
import pytest
import torch

from test_gpu_batch import problems, relerr   # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "mixed"])
def test_every_kernel_is_timed(bls, problems, dtype, monkeypatch):   # noqa: F811
    B = bls.batch.BatchedReduction(problems, dtype)
    assert B.run()
    S0, g0 = B.S.double().cpu().numpy(), B.g.cpu().numpy()
    ran = []
    run = B.run

    def counted(sync=True):
        ran.append((B.ws.phase2_kernel_name(dtype).split("<")[0], unit[0]))
        return run(sync)

    unit = [None]
    set_unit = B.ws.set_stage_unit
    monkeypatch.setattr(B, "run", counted)
    monkeypatch.setattr(B.ws, "set_stage_unit", lambda u: (unit.__setitem__(0, u), set_unit(u)))
    times = B.autotune(reps=2)
    kernels = {k for k, _ in ran}
    assert kernels == {"k_runs", "k_stage36", "k_pairs36"}, kernels
    assert {u for k, u in ran if k == "k_stage36"} == set(B.STAGE_UNITS)
    assert set(times) == {f"stage/{u}" for u in B.STAGE_UNITS} | {"pairs"}
    want = {"runs": "k_runs", "gather": "k_stage36", "pairs": "k_pairs36"}[B.kernel]
    assert B.ws.phase2_kernel_name(dtype).startswith(want)
    assert B.schedule == ("pairs" if B.kernel == "pairs" else "stage")
    for kernel in ("runs", "gather", "pairs", B.kernel):
        B.ws.set_kernel(kernel)
        assert run()
        assert relerr(B.S.double().cpu().numpy(), S0) <= (1e-12 if dtype == torch.float64 else 1e-6), kernel
        assert relerr(B.g.cpu().numpy(), g0) <= 1e-12, kernel
