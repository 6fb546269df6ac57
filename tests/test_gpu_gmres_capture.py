"""esr_gmres_cycle in a CUDA graph, in both its forms: replays advance the
solve as calls do, bit for bit."""
import numpy as np
import pytest
import torch

from easier_gb300.numeric.sparse import FusedGMRES, SellMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,one_launch", [(5000, True), (4_200_000, False)])
def test_captured_cycles(n, one_launch):
    i = np.arange(n - 1)
    row, col = np.concatenate([i, i + 1]), np.concatenate([i + 1, i])
    ae = torch.full((2 * (n - 1),), -1.0, dtype=torch.float64, device="cuda")
    A = SellMatrix.from_arrays(n, row, col, ae, torch.full((n,), 2.5, dtype=torch.float64, device="cuda"))
    eng = FusedGMRES(A, 3)
    assert eng.one_launch == one_launch
    b, x = torch.ones(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    r = torch.zeros_like(x)
    out = []
    for captured in (False, True):
        x.zero_()
        eng.solve(b, x, r, 0.0, None, 0)
        if captured:
            stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
                eng._cycle_call(b, x, r, 1)
            torch.cuda.current_stream().wait_stream(stream)
        for _ in range(3):
            graph.replay() if captured else eng._cycle_call(b, x, r, 1)
        assert eng.scalars().cycles == 3
        out.append(x.clone())
    assert torch.equal(*out)
