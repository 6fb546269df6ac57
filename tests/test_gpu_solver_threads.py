"""Two host threads that solve systems of different sizes with the cooperative
kernels: the launches of one may not depend on what the other asks for between
them (a kernel's shared-memory limit belongs to the function).  Both threads
launch into one stream, so the kernels themselves follow one another."""
import threading

import numpy as np
import pytest
import torch

from easier_gb300.numeric.batched import BatchedPCG, LinsysInstance
from easier_gb300.numeric.sparse import FusedGMRES, SellMatrix

pytestmark = pytest.mark.gpu


def _chain(n):
    """Tridiagonal, diagonally dominant."""
    i = np.arange(n - 1)
    row, col = np.concatenate([i, i + 1]), np.concatenate([i + 1, i])
    return LinsysInstance(n, row, col, np.full(2 * (n - 1), -1.0), np.full(n, 2.5), np.ones(n))


def _both(calls, count):
    errors = []

    def work(call):
        try:
            for _ in range(count):
                call()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[0]


def test_conjugate_gradients_of_two_sizes():
    engines = [BatchedPCG([_chain(n)], precision="fp64") for n in (900_000, 300_000)]  # both beyond 48 KB a CTA
    assert all(e.solo for e in engines)
    for e in engines:
        e.start(1e-10, None, None)
    _both([lambda e=e: e._solo_group(1) for e in engines], 2000)
    for e in engines:
        e.verify()
        assert e._info(e.instances()[0])["status"] == "converged"


def test_gmres_cycles_of_two_sizes():
    calls = []
    for n, restart in ((2_000_000, 4), (800_000, 4)):
        s = _chain(n)
        A = SellMatrix.from_arrays(n, s.row, s.col, torch.from_numpy(s.Ae).cuda(), torch.from_numpy(s.Av).cuda())
        eng = FusedGMRES(A, restart)
        assert eng.one_launch
        b, x = torch.ones(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
        r = torch.zeros_like(x)
        eng.solve(b, x, r, 0.0, None, 1)
        calls.append(lambda eng=eng, b=b, x=x, r=r: eng._cycle_call(b, x, r, 1))
    _both(calls, 500)


def test_solves_on_two_streams_at_once():
    """Two threads, a stream each: cooperative launches of either wait until
    all of their CTAs can run."""
    engines = [BatchedPCG([_chain(n)], precision="fp64") for n in (40_000, 60_000)]
    assert all(e.solo for e in engines)
    first = []
    for e in engines:
        info = e.solve(rtol=1e-10)
        first.append((info, e.solution(0).clone()))
    torch.cuda.synchronize()

    def solve(e, want, x, stream):
        with torch.cuda.stream(stream):
            e.reset()
            assert e.solve(rtol=1e-10) == want and torch.equal(e.solution(0), x)

    streams = [torch.cuda.Stream() for _ in engines]
    _both([lambda a=(e, *f, s): solve(*a) for e, f, s in zip(engines, first, streams)], 40)
