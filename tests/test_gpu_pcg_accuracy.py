"""The one-launch CG of an FP64 system is as accurate as the three-launch
iteration: distance of its iterate from CG in extended precision (numpy's long
double) after a fixed number of iterations, on the tutorial's finite-volume
Poisson systems without a preconditioner and on P1 grids with Jacobi.  Both
kernels round the same operations and differ in the order of their sums alone,
so over several right hand sides the distances agree: the geometric mean of
their ratio is held below 1.5 (the recurrence q = A z + beta q in place of
q = A p lies at 1.3 to 4)."""
import numpy as np
import pytest
import torch

from easier_gb300 import mesh
from easier_gb300.numeric.batched import BatchedPCG, LinsysInstance

pytestmark = pytest.mark.gpu


def _fv(n):
    m = mesh.triangular_mesh(n)
    a = mesh.poisson_fv(m)
    return [np.asarray(v) for v in (m.src, m.dst, a.Af, a.Ac)]


def _p1(n):
    s = mesh.p1_system(n)
    return [np.asarray(v) for v in (s.row, s.col, s.Ae, s.Av)]


def _extended(row, col, Ae, Av, b, jacobi, updates):
    n = b.shape[0]
    order = np.argsort(row, kind="stable")
    row, col, Ae = row[order], col[order], Ae[order].astype(np.longdouble)
    first = np.searchsorted(row, np.arange(n))
    diag = Av.astype(np.longdouble)
    inv = 1 / diag if jacobi else np.ones_like(diag)
    x, r = np.zeros(n, np.longdouble), b.astype(np.longdouble)
    p = z = inv * r
    rz = r @ z
    for _ in range(updates):
        q = np.add.reduceat(Ae * p[col], first) + diag * p
        a = rz / (p @ q)
        x, r = x + a * p, r - a * q
        z = inv * r
        new = r @ z
        p, rz = z + new / rz * p, new
    return x


@pytest.mark.parametrize("system,jacobi,iters", [(_fv(20), False, 130), (_fv(32), False, 210), (_p1(45), True, 125)])
def test_as_close_to_extended_precision_as_the_launch_sequence(system, jacobi, iters):
    row, col, Ae, Av = system
    n = Av.shape[0]
    ratios = []
    for seed in range(6):
        b = np.random.default_rng(seed).standard_normal(n) + 1.0
        exact = _extended(row, col, Ae, Av, b, jacobi, iters + 1)
        off = []
        for solo in (True, False):
            eng = BatchedPCG([LinsysInstance(n, row, col, Ae, Av, b)], jacobi=jacobi, precision="fp64")
            assert eng.solo
            eng.solo = solo
            info = eng.solve(rtol=0.0, maxiter=iters)[0]
            assert info["status"] == "maxiter" and info["iters"] == iters
            x = eng.solution(0).cpu().numpy().astype(np.longdouble)
            off.append(float(np.sqrt(((x - exact) ** 2).sum() / (exact ** 2).sum())))
        assert off[0] < 1e-13
        ratios.append(off[0] / off[1])
    assert np.exp(np.mean(np.log(ratios))) <= 1.5, ratios
