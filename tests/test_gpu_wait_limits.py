"""Waits between CTAs and warps that run out.  The entry points in which every
wait gives up at once stand in for the ordinary ones, so no wait takes long and
no GPU error is involved: the status bit, the solve's own mark, the Python
error, and that the next ordinary solve on the same engine is the first one's."""
import numpy as np
import pytest
import torch

from easier_gb300 import _lib, ops
from easier_gb300.numeric.batched import BatchedPCG, LinsysInstance
from easier_gb300.numeric.sparse import FusedGMRES, SellMatrix

pytestmark = pytest.mark.gpu

BOUNDED = ("esr_bcg_iterate", "esr_pcg_solo_iterate", "esr_gmres_cycles")


def _chain(n):
    i = np.arange(n - 1)
    row, col = np.concatenate([i, i + 1]), np.concatenate([i + 1, i])
    return LinsysInstance(n, row, col, np.full(2 * (n - 1), -1.0), np.full(n, 2.5), np.ones(n))


@pytest.fixture
def hurried(monkeypatch):
    """A context in which every bounded wait gives up at once."""
    call = _lib.call

    def patched(name, *args):
        call(name + "_timeout" if name in BOUNDED else name, *args)

    def run(f):
        ops.device_status(clear=True)
        with monkeypatch.context() as m:
            m.setattr(_lib, "call", patched)
            with pytest.raises(RuntimeError, match="timed out"):
                f()
        assert ops.device_status(clear=True) == _lib.DEV_WAIT_TIMEOUT

    return run


@pytest.mark.parametrize("n,jacobi", [(300, True), (5000, False), (200_000, True), (200_000, False)])
def test_one_launch_cg(n, jacobi, hurried):
    eng = BatchedPCG([_chain(n)], jacobi=jacobi, precision="fp64")
    assert eng.solo
    first, x = eng.solve(rtol=1e-9), eng.solution(0).clone()
    eng.reset()
    hurried(lambda: eng.solve(rtol=1e-9))
    assert eng.instances()[0].done == 4 and eng.active() == 0
    eng.reset()  # (the mailboxes were zeroed)
    assert eng.solve(rtol=1e-9) == first and torch.equal(eng.solution(0), x)


@pytest.mark.parametrize("precision", ["df64", "fp64"])
def test_streamed_sweeps(precision, hurried):
    eng = BatchedPCG([_chain(n) for n in (300, 5000, 256)], precision=precision, use_graph=False)
    eng.set_shape(1, 4)
    first, x = eng.solve(rtol=1e-9), eng.solution().clone()
    eng.reset()
    hurried(lambda: eng.solve(rtol=1e-9))
    assert all(s.done == 4 for s in eng.instances()) and eng.active() == 0
    eng.reset()
    assert eng.solve(rtol=1e-9) == first and torch.equal(eng.solution(), x)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,restart", [(300, 5), (40_000, 20)])
def test_gmres_cycles(n, restart, dtype, hurried):
    s = _chain(n)
    A = SellMatrix.from_arrays(n, s.row, s.col, torch.from_numpy(s.Ae).cuda(), torch.from_numpy(s.Av).cuda(), dtype)
    eng = FusedGMRES(A, restart)
    assert eng.one_launch
    b, x = torch.ones(n, dtype=dtype, device="cuda"), torch.zeros(n, dtype=dtype, device="cuda")
    r = torch.zeros_like(x)
    eng.solve(b, x, r, 1e-5, None, 20)
    good = x.clone()
    x.zero_()
    hurried(lambda: eng.solve(b, x, r, 1e-5, None, 20))
    x.zero_()
    eng.solve(b, x, r, 1e-5, None, 20)
    assert torch.equal(x, good)
