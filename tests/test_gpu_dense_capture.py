"""DenseCholesky.solve inside a CUDA graph: the waits between its tiles and its memset replay with it. Tolerance 1e-10
relative as in test_gpu_dense.py."""
import numpy as np
import pytest
import torch

from test_gpu_dense import relerr
from test_gpu_dense_tiles import spd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 700])
def test_solve_in_a_graph(bls, n):
    A, rng = spd(n, 13)
    D = bls.DenseCholesky(n)
    assert D.factor(torch.from_numpy(np.triu(A).ravel(order="F")).to("cuda"))
    g, x = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.cuda.graph(graph, stream=side):
        D.solve(g, x)
        D.solve(x, x)
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(3):
        b = rng.standard_normal(n)
        g.copy_(torch.from_numpy(b))
        graph.replay()
        assert relerr(x.cpu().numpy(), np.linalg.solve(A, np.linalg.solve(A, b))) <= 1e-10
    graph.reset()
