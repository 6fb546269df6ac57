"""What the solvers do with a wait that gave up on the device and with the
device's status bits: a time-out is the solve's own (done = 4, GMRES's
broken = 2) and raises; an ordinary breakdown is no time-out, whatever bits
other calls have raised, and leaves those bits to whoever asks for them."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from easier_gb300 import _lib, ops
from easier_gb300.numeric.batched import BatchedPCG, LinsysInstance
from easier_gb300.numeric.sparse import FusedGMRES


def _engine(monkeypatch):
    def asked(*a, **k):
        raise AssertionError("a solve reads (and clears) the device's status bits")

    monkeypatch.setattr(ops, "device_status", asked)
    eng = object.__new__(BatchedPCG)
    eng.solo, eng._solo_comm = True, torch.ones(8, dtype=torch.uint8)
    return eng


def test_a_breakdown_leaves_the_status_bits_alone(monkeypatch):
    eng = _engine(monkeypatch)
    insts = [SimpleNamespace(done=1), SimpleNamespace(done=3)]
    assert eng._checked(insts) is insts
    assert int(eng._solo_comm.sum()) == 8


def test_a_timed_out_instance_raises_and_its_mailboxes_are_cleared(monkeypatch):
    eng = _engine(monkeypatch)
    with pytest.raises(RuntimeError, match="timed out"):
        eng._checked([SimpleNamespace(done=1), SimpleNamespace(done=4)])
    assert int(eng._solo_comm.sum()) == 0


def test_a_timed_out_gmres_cycle_raises(monkeypatch):
    eng = object.__new__(FusedGMRES)
    eng.A, eng.dev, eng.ws, eng.kernel_launches, eng.one_launch = SimpleNamespace(desc=_lib.Sell()), None, None, 0, True
    states = iter([SimpleNamespace(cycles=0, broken=0, rnorm=1.0, tol=1e-9), SimpleNamespace(cycles=1, broken=2, rnorm=float("nan"), tol=1e-9)])
    monkeypatch.setattr(_lib, "call", lambda *a: None)
    monkeypatch.setattr(_lib, "stream_handle", lambda *a: 0)
    monkeypatch.setattr(_lib, "ptr", lambda t: 0)
    eng.scalars = lambda: next(states)
    eng._cycle = lambda *a: None
    with pytest.raises(RuntimeError, match="timed out"):
        eng.solve(None, None, None, 1e-9, None, None)


@pytest.mark.gpu
@pytest.mark.parametrize("count,precision", [(1, "fp64"), (1, "df64"), (2, "fp64")])
def test_pending_bits_survive_a_breakdown_of_another_solve(count, precision):
    ops.device_status(clear=True)
    x, y = torch.zeros(4, device="cuda"), torch.zeros(1, device="cuda")
    idx = torch.tensor([9], dtype=torch.int32, device="cuda")  # (checked by the kernel)
    _lib.call("esr_gather", x.data_ptr(), 4, 4, idx.data_ptr(), 1, y.data_ptr(), _lib.stream_handle())
    gave_up = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("esr_wait_selftest", 16, gave_up.data_ptr(), _lib.stream_handle())
    row, col = np.array([0, 1]), np.array([1, 0])
    b = np.ones(300)
    b[7] = np.nan
    inst = LinsysInstance(300, row, col, np.full(2, -0.5), np.full(300, 2.0), b)
    info = BatchedPCG([inst] * count, precision=precision).solve(rtol=1e-9, maxiter=50)
    assert all(i["status"] == "breakdown" for i in info)
    assert ops.device_status(clear=True) == _lib.DEV_IDX_RANGE | _lib.DEV_WAIT_TIMEOUT
