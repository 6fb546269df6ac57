"""Selector, Reducer, Linsys and aggregator kernels at the sizes where their
tiling can go wrong: tile edges, remainders, long segments, wide rows, every
dispatch branch.  Bitwise against the oracle (order-fixed work) or the
op-by-op path; sums within the rounding bound n * 2^-53 * sum |x|."""
import numpy as np
import pytest
import torch

import easier_gb300 as esr
from easier_gb300 import _lib, ops
from easier_gb300.numeric import Linsys
from oracle import sparse as osp

pytestmark = pytest.mark.gpu


def _module(sel=None, red=None, n=0, op="sum"):
    class M(esr.Module):
        def __init__(self):
            super().__init__()
            if sel is not None:
                self.sel = esr.Selector(sel)
            if red is not None:
                self.red = esr.Reducer(red, n, op)
    m = M()
    esr.compile([m], "cuda")
    return m


@pytest.mark.parametrize("m", [1, 255, 257, 1025, 1_300_000])
@pytest.mark.parametrize("dtype,tail", [(torch.uint8, (3,)), (torch.float32, ()), (torch.float32, (3,)),
                                        (torch.float64, (3,)), (torch.float32, (4,)), (torch.int64, (7,))])
def test_gather_tiles(m, dtype, tail):
    g = torch.Generator().manual_seed(m)
    n = 1000
    idx = torch.randint(0, n, (m,), generator=g)
    x = torch.randint(0, 200, (n,) + tail, generator=g).to(dtype)
    assert torch.equal(_module(sel=idx).sel(x.cuda()).cpu(), x[idx])


@pytest.mark.parametrize("cols", [1023, 1024, 1025, 4100])
def test_gather_wide_rows(cols):
    g = torch.Generator().manual_seed(cols)
    idx = torch.randint(0, 37, (50,), generator=g)
    x = torch.randn(37, cols, generator=g)
    mod = _module(sel=idx)
    assert torch.equal(mod.sel(x.cuda()).cpu(), x[idx])
    y = torch.randn(37, cols + 1, generator=g)[:, 1:].contiguous()  # odd 4-byte offsets
    flat = torch.cat([torch.zeros(1), y.reshape(-1)]).cuda()[1:].view(37, cols)
    assert torch.equal(mod.sel(flat).cpu(), y[idx])


@pytest.mark.parametrize("op", ["sum", "mean", "prod", "amax", "amin"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.int64])
@pytest.mark.parametrize("cols", [1, 2, 3, 5, 255, 256, 257])
def test_segments(op, dtype, cols):
    """Rows without entries, rows longer than a staged chunk, a last tile cut
    short; sorted indices (no permutation) and shuffled ones."""
    if op in ("mean", "prod") and not dtype.is_floating_point:
        pytest.skip("floating reductions")
    g = torch.Generator().manual_seed(cols)
    n = 301 if cols < 100 else 7
    long = torch.full((2500,), 2) if cols < 100 else torch.full((40,), 2)
    idx = torch.cat([torch.randint(0, n - 2, (900 if cols < 100 else 60,), generator=g), long])
    idx[idx == 4] = 5  # row 4 and the last row stay empty
    for shuffled in (False, True):
        i = idx[torch.randperm(idx.shape[0], generator=g)] if shuffled else idx.sort().values
        t = torch.randn(i.shape[0], *(() if cols == 1 else (cols,)), generator=g, dtype=torch.float64)
        t = (t if dtype.is_floating_point else t * 1000).to(dtype)
        if dtype.is_floating_point:
            t[3] = -0.0
            if op.startswith("a"):
                t[7] = float("nan")
                t[9] = float("inf")
        mod = _module(red=i, n=n, op=op)
        assert mod.red._in_row_order == (not shuffled)
        got, want = mod.red(t.cuda()).cpu(), osp.reduce(t, i, n, op)
        assert np.array_equal(got.numpy(), want.numpy(), equal_nan=dtype.is_floating_point)
        out = torch.full_like(want, 3)
        kept = mod.red(t.cuda(), out=out.cuda()).cpu()
        empty = torch.bincount(i, minlength=n) == 0
        assert torch.equal(kept[empty], out[empty]) and int(empty.sum()) >= 2
        assert np.array_equal(kept[~empty].numpy(), want[~empty].numpy(), equal_nan=dtype.is_floating_point)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,m,shuffled", [(1, 0, False), (255, 900, True), (256, 2048, False), (257, 5001, True),
                                          (70_001, 400_000, True)])
def test_linsys_apply_is_bitwise_the_five_operations(dtype, n, m, shuffled):
    g = torch.Generator().manual_seed(n)
    row = torch.randint(0, n, (m,), generator=g)
    row = row if shuffled else row.sort().values
    col = torch.randint(0, n, (m,), generator=g)

    class M(esr.Module):
        def __init__(self):
            super().__init__()
            self.sel, self.red = esr.Selector(col), esr.Reducer(row, n)
            self.Ae = esr.Tensor(torch.randn(m, generator=g).to(dtype), mode="partition")
            self.Av = esr.Tensor(torch.randn(n, generator=g).to(dtype), mode="partition")
            self.A = Linsys(self.Av, self.Ae, self.sel, self.red)

    mod = M()
    esr.compile([mod], "cuda")
    x = torch.randn(n, generator=g).to(dtype)
    x[n // 2] = -0.0
    wide = torch.stack([x, x], 1).cuda()
    for v in (x.cuda(), wide[:, 0]):  # contiguous and strided
        fused = ops.linsys_apply(mod.A, v)
        assert fused is not None
        want = mod.red(mod.sel(v) * mod.Ae) + v * mod.Av
        assert torch.equal(fused, want) and torch.equal(mod.A(v), want)
    if m and dtype == torch.float64:
        bad = x.cuda()
        bad[0] = float("inf")
        want = mod.red(mod.sel(bad) * mod.Ae) + bad * mod.Av
        assert np.array_equal(mod.A(bad).cpu().numpy(), want.cpu().numpy(), equal_nan=True)
        # what the kernel does not cover keeps the five operations
        assert ops.linsys_apply(mod.A, x.float().cuda()) is None
        assert mod.A(x.float().cuda()).dtype == torch.float64
        v = x.cuda().requires_grad_()
        assert ops.linsys_apply(mod.A, v) is None and mod.A(v).requires_grad


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.int32, torch.int64])
@pytest.mark.parametrize("n,cols", [(1, 1), (8192, 1), (8193, 1), (1_000_003, 1), (5000, 2), (40_001, 3), (300, 64),
                                    (2049, 255), (777, 256), (777, 257), (9, 1000)])
def test_aggregates(dtype, n, cols):
    g = torch.Generator().manual_seed(n + cols)
    t = torch.randn(n, *(() if cols == 1 else (cols,)), generator=g, dtype=torch.float64)
    t = (t if dtype.is_floating_point else t * 1000).to(dtype)
    c, d = t.cuda(), t.double()
    assert torch.equal(esr.max(c).cpu(), t.amax(0, keepdim=True))
    assert torch.equal(esr.min(c).cpu(), t.amin(0, keepdim=True))
    if not dtype.is_floating_point:
        assert torch.equal(esr.sum(c).cpu(), t.sum(0, keepdim=True).to(dtype))
        return
    ulp = torch.finfo(dtype).eps
    bound = n * 2.0 ** -53 * d.abs().sum(0, keepdim=True)
    want = d.sum(0, keepdim=True)
    assert bool(((esr.sum(c).cpu().double() - want).abs() <= bound + ulp * want.abs()).all())
    want = d.norm(dim=0, keepdim=True)
    assert bool(((esr.norm(c).cpu().double() - want).abs() <= (n * 2.0 ** -53 + 2 * ulp) * want).all())
    assert torch.equal(esr.sum(c), esr.sum(c))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_extrema_of_special_values(dtype):
    lo, hi = -torch.finfo(dtype).max, torch.finfo(dtype).max
    inf, nan = float("inf"), float("nan")
    for vals, mx, mn in (([-inf, -inf], -inf, -inf), ([lo, -inf], lo, -inf), ([inf, hi], inf, hi), ([-1.0, nan], nan, nan),
                         ([-nan, 2.0], nan, nan), ([-0.0, -0.0], 0.0, 0.0), ([5e-45, -5e-45], 5e-45, -5e-45)):
        for n in (2, 20_000):
            t = torch.tensor(vals, dtype=dtype).repeat(n // 2).cuda()
            for got, want in ((esr.max(t), mx), (esr.min(t), mn)):
                want = torch.tensor([want], dtype=dtype)
                assert np.array_equal(got.cpu().numpy(), want.numpy(), equal_nan=True), (vals, n)


def test_empty_aggregates():
    t = torch.zeros(0, 3, dtype=torch.float64, device="cuda")
    assert torch.equal(esr.sum(t).cpu(), torch.zeros(1, 3, dtype=torch.float64))
    assert torch.equal(ops.aggregate(t, "prod").cpu(), torch.ones(1, 3, dtype=torch.float64))
    assert ops.device_status(clear=True) & _lib.DEV_IDX_RANGE == 0
