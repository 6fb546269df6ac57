"""The streamed sweeps of the batched PCG where their copies and sums can go
wrong: slices of every width (also wider than a stage holds), instances at the
edges of a tile, chunks of one tile, more chunks a CTA than a warp reads heads
of at once, and buffers that begin off the 16 bytes the bulk copies need."""
import numpy as np
import pytest
import torch

from easier_gb300.numeric.batched import BatchedPCG, LinsysInstance

pytestmark = pytest.mark.gpu


def _ring(n, reach, seed):
    """Symmetric and diagonally dominant, `2 reach` couplings a row (fewer where
    n is too small for them to differ)."""
    rng = np.random.default_rng(seed)
    dense = np.zeros((n, n))
    for d in range(1, reach + 1):
        w = -rng.uniform(0.2, 1.0, n)
        for i in range(n):
            j = (i + d) % n
            if i != j:
                dense[i, j] = dense[j, i] = w[i]
    diag = -dense.sum(axis=1) + rng.uniform(0.5, 1.0, n)
    row, col = np.nonzero(dense)
    inst = LinsysInstance(n, row, col, dense[row, col], diag, rng.uniform(-1.0, 1.0, n))
    return inst, dense + np.diag(diag)


def _solved(eng, mats, insts):
    # the solver's own stopping test, on the FP64 residual
    for i, (m, s) in enumerate(zip(mats, insts)):
        x = eng.solution(i).cpu().numpy()
        assert np.linalg.norm(s.b - m @ x) <= 1.0001e-9 * np.linalg.norm(s.b), i


@pytest.mark.parametrize("precision", ["df64", "fp64"])
@pytest.mark.parametrize("reach", [1, 2, 3, 4, 5, 20])
def test_every_slice_width_and_tile_edge(precision, reach):
    pairs = [_ring(n, reach, 7 * n + reach) for n in (2, 31, 255, 256, 257, 600)]
    insts, mats = [p[0] for p in pairs], [p[1] for p in pairs]
    eng = BatchedPCG(insts, precision=precision)
    ref = None
    for tiles, grid in ((1, 1), (1, 500), (2, 3)):
        eng.set_shape(tiles, grid)
        eng.reset()
        res = eng.solve(rtol=1e-9)
        assert all(r["status"] == "converged" for r in res)
        _solved(eng, mats, insts)
        x = eng.solution().clone()
        if tiles == 1:  # the same chunks, whatever CTA takes them: the same bits
            assert ref is None or torch.equal(x, ref)
            ref = x


@pytest.mark.parametrize("precision", ["df64", "fp64"])
def test_more_chunks_than_heads_and_odd_buffers(precision):
    inst, mat = _ring(1400, 2, 3)
    insts, mats = [inst] * 8, [mat] * 8  # 48 tiles
    eng = BatchedPCG(insts, precision=precision)
    eng.set_shape(1, 1)
    res = eng.solve(rtol=1e-9)
    assert all(r["status"] == "converged" for r in res)
    _solved(eng, mats, insts)
    x = eng.solution().clone()
    for name in ("x", "r", "z", "p", "q"):  # 8 bytes into their storage
        t = getattr(eng, name)
        flat = torch.zeros(t.numel() + 4, dtype=t.dtype, device=t.device)
        off = 8 // t.element_size()
        setattr(eng, name, flat[off:off + t.numel()].view(t.shape))
    assert eng.x.data_ptr() % 16 == 8
    eng.set_shape(1, 1)  # (no captured launches on the old buffers)
    again = eng.solve(rtol=1e-9)
    assert [r["iters"] for r in again] == [r["iters"] for r in res]
    assert torch.equal(eng.solution(), x)
