"""The one-launch GMRES cycle against the per-operation loop over every form it
takes: row counts around slices and CTAs, one to 64 columns (sums formed one
or two a warp), the basis on the chip and off it, FP64 and FP32, every way a
solve can end, launches of any number of cycles; and the launch sequence that
larger systems keep."""
import numpy as np
import pytest
import torch

import easier_gb300 as esr
from easier_gb300.numeric import Linsys, sparse
from easier_gb300.numeric.preconditioner import Jacobi
from easier_gb300.numeric.solver import GMRES

pytestmark = pytest.mark.gpu


class _System(esr.Module):
    """Unsymmetric, diagonally dominant, some of the couplings in one wide row."""

    def __init__(self, n, degree=4, seed=0, dtype=torch.float64, diag=None, b=None):
        super().__init__()
        g = np.random.default_rng(seed)
        m = max(n * degree, 1)
        row, col = g.integers(0, n, m), g.integers(0, n, m)
        if n > 40:
            row[:12] = 7
        val = g.standard_normal(m)
        if diag is not None:  # diag * I (with one coupling that adds nothing: a Linsys has some)
            val = np.where(np.arange(m) == 0, 1e-300, 0.0)
        d = np.bincount(row, weights=np.abs(val), minlength=n) * 1.05 + 0.1 if diag is None else np.full(n, diag)
        t = torch.from_numpy
        self.red, self.sel = esr.Reducer(t(row), n), esr.Selector(t(col))
        self.Ae, self.Av = esr.Tensor(t(val), mode="partition"), esr.Tensor(t(d), mode="partition")
        self.b = esr.Tensor(t(g.standard_normal(n) if b is None else b), mode="partition")
        self.x = esr.Tensor(esr.zeros((n,), dtype=torch.float64), mode="partition")
        self.A = Linsys(self.Av, self.Ae, self.sel, self.red)
        self.to("cuda")
        if dtype != torch.float64:
            self.to(dtype)


def _solver(sysm, restart, jacobi=True):
    sol = GMRES(sysm.A, sysm.b, sysm.x, M=Jacobi(sysm.A) if jacobi else None, restart=restart)
    esr.compile([sysm, sol], "cuda")
    return sol


def _residual(s):
    x, b = s.x.data.double(), s.b.data.double()
    ax = torch.zeros_like(x).index_add_(0, s.red.idx, x[s.sel.idx] * s.Ae.data.double()) + x * s.Av.data.double()
    return float((b - ax).norm() / b.norm())


@pytest.mark.parametrize("n,restart,jacobi", [(1, 1, True), (31, 5, False), (33, 16, True), (257, 17, True),
                                              (4097, 33, False), (4097, 2, True), (40_000, 20, True),
                                              (90_001, 64, False), (300_000, 24, True)])
def test_cycles_as_the_per_operation_loop(n, restart, jacobi):
    fused, loop = _System(n, seed=n), _System(n, seed=n)
    a, b = _solver(fused, restart, jacobi), _solver(loop, restart, jacobi)
    ia, ib = a.solve(rtol=1e-10, maxiter=200), b.solve(rtol=1e-10, maxiter=200, fused=False)
    assert a._fused.one_launch
    assert abs(ia["iters"] - ib["iters"]) <= 1
    assert _residual(fused) <= 1.01e-10 and _residual(loop) <= 1.01e-10
    # a fixed number of cycles: the same minimisation, so the same iterate
    for s, sol, kw in ((fused, a, {}), (loop, b, dict(fused=False))):
        s.x[:] = 0.0
        sol.solve(rtol=0.0, maxiter=2, **kw)
    # (two cycles from zero amplify rounding by at most the residual's reduction)
    assert float((fused.x.data - loop.x.data).norm()) <= 1e-8 * float(loop.x.data.norm())


def test_fp32():
    s, ref = _System(5000, seed=3, dtype=torch.float32), _System(5000, seed=3, dtype=torch.float32)
    sol, per_op = _solver(s, 20), _solver(ref, 20)
    a, b = sol.solve(rtol=1e-5, maxiter=50), per_op.solve(rtol=1e-5, maxiter=50, fused=False)
    assert abs(a["iters"] - b["iters"]) <= 1 and _residual(s) <= 2e-5


def test_endings():
    s = _System(3000, seed=1)
    sol = _solver(s, 10)
    assert sol.solve(rtol=1e-10, maxiter=0)["iters"] == 0
    assert sol.solve(rtol=1e-30, maxiter=3)["iters"] == 3
    done = sol.solve(rtol=1e-10)
    assert _residual(s) <= 1.01e-10 and done["iters"] >= 1
    assert sol.solve(rtol=1e-9)["iters"] == 0  # already there
    # a Krylov space of one dimension: the cycle runs out of it and has the solution
    one = _System(500, seed=2, diag=3.0)
    sol = _solver(one, 8, jacobi=False)
    assert sol.solve(rtol=1e-12, maxiter=5)["iters"] == 1
    assert torch.allclose(one.x.data, one.b.data / 3.0, rtol=1e-13)
    zero = _System(500, seed=2, b=np.zeros(500))
    assert _solver(zero, 8).solve(rtol=1e-10, maxiter=5) == {"residual": 0.0, "iters": 0}
    bad = np.ones(500)
    bad[3] = np.nan
    info = _solver(_System(500, seed=2, b=bad), 8).solve(rtol=1e-10, maxiter=5)
    assert info["iters"] == 5 and np.isnan(info["residual"])


def test_launches_of_any_number_of_cycles_give_the_same_bits(monkeypatch):
    out = []
    for most in (16, 3, 1):
        monkeypatch.setattr(sparse, "GMRES_CYCLES", most)
        s = _System(6000, seed=8)
        info = _solver(s, 3).solve(rtol=1e-9, maxiter=100)
        out.append((info["iters"], info["residual"], s.x.data.clone()))
    for it, res, x in out[1:]:
        assert it == out[0][0] and res == out[0][1] and torch.equal(x, out[0][2])


def test_larger_systems_keep_the_launch_sequence():
    s = _System(4_200_000, degree=2, seed=4)
    sol = _solver(s, 5)
    assert sol.solve(rtol=1e-6, maxiter=60)["iters"] < 60
    assert not sol._fused.one_launch and _residual(s) <= 1.01e-6
