"""FP64 steps of small meshes, which take a lane a face, against the same RK4
step put together from the delta kernel (a thread a cell) by torch, bit for bit:
cells at the edges of a warp's and a CTA's share, three and four face slots,
walls, empty slots, and both sides of the size where the launch changes."""
import ctypes

import pytest
import torch

from easier_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [3, 4])
@pytest.mark.parametrize("nc", [1, 7, 8, 9, 10, 11, 31, 32, 39, 40, 41, 1000, 100000, 100001])
def test_steps_equal_delta_kernel_steps_bitwise(width, nc):
    g = torch.Generator(device="cuda").manual_seed(31 * nc + width)
    rnd = lambda *s: torch.rand(s, generator=g, dtype=torch.float64, device="cuda")
    nbr = torch.randint(-2, nc, (width, nc), generator=g, device="cuda", dtype=torch.int32)
    nbr[0] = torch.where(rnd(nc) < 0.5, nbr[0], nbr[0].clamp(min=0))
    sx, sy = rnd(width, nc) - 0.5, rnd(width, nc) - 0.5
    sx[:, ::3] = 0.0  # (faces along an axis)
    sy[:, 1::5] = 0.0
    alpha, area = rnd(width, nc), 0.5 + rnd(nc)
    state = torch.zeros(nc, 4, dtype=torch.float64, device="cuda")
    state[:, 0] = 0.5 + rnd(nc)
    state[:, 1:3] = rnd(nc, 2) - 0.5
    state[::2, 1:3] = 0.0  # water at rest
    mesh = _lib.SweMesh(nc, width, _lib.dtype_code(torch.float64), _lib.ptr(nbr), _lib.ptr(sx), _lib.ptr(sy),
                        _lib.ptr(alpha), _lib.ptr(area), _lib.ptr(area), 1, 0)
    ws = torch.empty(int(_lib.lib().esr_swe_workspace_bytes(ctypes.byref(mesh))), dtype=torch.uint8, device="cuda")
    stream = _lib.stream_handle(torch.device("cuda"))
    dt = 1e-3

    def delta(s):
        out = torch.empty_like(s)
        _lib.call("esr_swe_delta", ctypes.byref(mesh), _lib.ptr(s), _lib.ptr(out), stream)
        return out

    want = state.clone()
    for _ in range(2):
        k1 = delta(want)
        k2 = delta(want + (0.5 * dt) * k1)
        k3 = delta(want + (0.5 * dt) * k2)
        k4 = delta(want + dt * k3)
        want = want + (dt / 6) * ((((k1 + k2) + k3)) + k4)
    _lib.call("esr_swe_step", ctypes.byref(mesh), dt, _lib.ptr(state), 2, _lib.ptr(ws), stream)
    assert torch.isfinite(want).all()
    assert torch.equal(state, want)
