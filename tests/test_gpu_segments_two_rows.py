"""Segment sums with two rows a thread (from 622,592 rows up): rows around the
last CTA's two halves, empty rows, rows longer than the entries a thread loads
at once; bitwise the oracle's, with and without `out`."""
import numpy as np
import pytest
import torch

import easier_gb300 as esr
from oracle import sparse as osp

pytestmark = pytest.mark.gpu

TWO_ROWS = 152 * 8 * 2 * 256


@pytest.mark.parametrize("n", [TWO_ROWS - 1, TWO_ROWS, TWO_ROWS + 255, TWO_ROWS + 300])
@pytest.mark.parametrize("op,dtype,cols,shuffled", [("sum", torch.float32, 3, True), ("sum", torch.float64, 1, False),
                                                    ("mean", torch.float64, 2, True), ("amax", torch.float32, 4, True),
                                                    ("amin", torch.float64, 1, True), ("sum", torch.int64, 2, False)])
def test_two_rows_a_thread(n, op, dtype, cols, shuffled):
    g = torch.Generator().manual_seed(n + cols)
    idx = torch.cat([torch.randint(0, n, (700_000,), generator=g), torch.full((9,), n - 2), torch.full((9,), n - 257)])
    idx = idx[(idx != n - 1) & (idx != 5)]  # two rows stay empty (others too)
    if not shuffled:
        idx = idx.sort().values
    t = torch.randn(idx.shape[0], *(() if cols == 1 else (cols,)), generator=g, dtype=torch.float64)
    t = (t if dtype.is_floating_point else t * 1000).to(dtype)

    class M(esr.Module):
        def __init__(self):
            super().__init__()
            self.red = esr.Reducer(idx, n, op)

    mod = M()
    esr.compile([mod], "cuda")
    want = osp.reduce(t, idx, n, op)
    assert np.array_equal(mod.red(t.cuda()).cpu().numpy(), want.numpy())
    out = torch.full_like(want, 3)
    empty = torch.bincount(idx, minlength=n) == 0
    kept = mod.red(t.cuda(), out=out.cuda()).cpu()
    assert int(empty.sum()) >= 2 and torch.equal(kept[empty], out[empty]) and torch.equal(kept[~empty], want[~empty])
