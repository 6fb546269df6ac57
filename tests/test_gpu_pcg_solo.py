"""The one-launch CG of a single FP64 system against the three-launch
iteration of the batched engine, over every form its rule accepts: row counts
around slices and CTAs, rows wider than its unrolled widths, with and without
Jacobi, every way a solve can end, and launches cut at any iteration."""
import numpy as np
import pytest
import torch

from easier_gb300.numeric import batched
from easier_gb300.numeric.batched import BatchedPCG, LinsysInstance

pytestmark = pytest.mark.gpu


def _system(n, degree, seed):
    """Symmetric, diagonally dominant, about `degree` couplings a row, some of
    them in one much wider row."""
    g = np.random.default_rng(seed)
    m = n * degree // 2
    i, j = g.integers(0, n, m), g.integers(0, n, m)
    if n > 40:
        i[:12], j[:12] = 7, np.arange(20, 32)  # row 7: beyond eight slots
    keep = i != j
    i, j = i[keep], j[keep]
    v = -g.random(i.shape[0])
    row, col, val = np.concatenate([i, j]), np.concatenate([j, i]), np.concatenate([v, v])
    diag = np.bincount(row, weights=-val, minlength=n) + 0.05 + g.random(n)
    return LinsysInstance(n, row, col, val, diag, g.standard_normal(n))


def _pair(inst, jacobi):
    solo, multi = (BatchedPCG([inst], jacobi=jacobi, precision="fp64") for _ in range(2))
    assert solo.solo
    multi.solo = False
    return solo, multi


@pytest.mark.parametrize("jacobi", [True, False])
@pytest.mark.parametrize("n,degree", [(3, 8), (31, 2), (32, 3), (257, 4), (600, 6), (4097, 3), (4096, 11), (40_000, 4),
                                      (90_001, 4)])
def test_solves_as_the_multi_launch_engine(n, degree, jacobi):
    inst = _system(n, degree, n)
    solo, multi = _pair(inst, jacobi)
    a, b = (e.solve(rtol=1e-10)[0] for e in (solo, multi))
    assert a["status"] == b["status"] == "converged" and abs(a["iters"] - b["iters"]) <= 1
    assert a["true_residual"] <= a["tol"]
    x, y = solo.solution(0), multi.solution(0)
    assert float((x - y).norm()) <= 1e-8 * float(y.norm())  # both within rtol of the same solution
    assert np.isclose(a["bnorm"], b["bnorm"], rtol=1e-13)


@pytest.mark.parametrize("jacobi", [True, False])
def test_every_ending_is_the_multi_launch_engines(jacobi):
    inst = _system(3000, 4, 5)
    solo, multi = _pair(inst, jacobi)
    x_true = multi.solution(0).clone()

    def both(b=None, x0=None, **kw):
        out = []
        for e in (solo, multi):
            e.load_instance(0, b=torch.as_tensor(inst.b if b is None else b),
                            x0=torch.zeros(3000, dtype=torch.float64) if x0 is None else x0)
            out.append(e.solve(**kw)[0])
        return out

    for kw in (dict(rtol=1e-10, maxiter=0), dict(rtol=1e-10, maxiter=1), dict(rtol=1e-10, maxiter=7),
               dict(rtol=0.0, atol=1e-3), dict(rtol=10.0), dict(rtol=1e-10, b=np.zeros(3000)),
               dict(rtol=1e-10, b=np.where(np.arange(3000) == 5, np.nan, inst.b)),
               dict(rtol=1e-10, b=np.where(np.arange(3000) == 5, np.inf, inst.b))):
        a, b = both(**kw)
        assert (a["status"], a["iters"]) == (b["status"], b["iters"]), kw
        if a["status"] == "converged":  # (after many iterations the two roundings have drifted apart)
            assert a["residual"] <= a["tol"] and b["residual"] <= b["tol"], kw
        else:
            assert np.isclose(a["residual"], b["residual"], rtol=1e-9, atol=1e-300, equal_nan=True), kw
    # a residual replacement: b changes under a converged recurrence
    for e in (solo, multi):
        e.load_instance(0, b=torch.as_tensor(inst.b), x0=x_true)
        e.start(1e-10, None, None)
        (e._solo_group if e.solo else e._group)(64)
        e.load_instance(0, b=torch.as_tensor(inst.b) * 1.5)
        while True:
            e.verify()
            if e.active() == 0:
                break
            while e.active():
                (e._solo_group if e.solo else e._group)(32)
        info = e._info(e.instances()[0])
        assert info["status"] == "converged" and info["restarts"] >= 1


def test_cut_launches_give_the_same_bits(monkeypatch):
    inst = _system(5000, 4, 9)
    results = []
    for most in (4096, 5, 1):
        monkeypatch.setattr(batched, "SOLO_ITERS", most)
        eng = BatchedPCG([inst], precision="fp64")
        info = eng.solve(rtol=1e-10)[0]
        results.append((info["iters"], info["residual"], eng.solution(0).clone()))
    for iters, residual, x in results[1:]:
        assert iters == results[0][0] and residual == results[0][1] and torch.equal(x, results[0][2])


def test_what_does_not_qualify_keeps_the_multi_launch_engine():
    inst = _system(500, 4, 1)
    assert not BatchedPCG([inst, inst], precision="fp64").solo
    assert not BatchedPCG([inst], precision="df64").solo
    assert not BatchedPCG([inst], precision="fp64", poly_degree=2).solo
    big = LinsysInstance(1_300_000, np.array([0, 1]), np.array([1, 0]), np.full(2, -0.5), np.full(1_300_000, 2.0),
                         np.ones(1_300_000))
    eng = BatchedPCG([big], precision="fp64")
    assert not eng.solo and eng.solve(rtol=1e-10)[0]["status"] == "converged"
