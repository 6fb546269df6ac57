"""Device ops behind Selector / Reducer / aggregators.

Each op checks its inputs on the host (device, dtype, shape, index range
known since compile) and launches the matching C-ABI kernel on torch's
current stream.  Non-CUDA tensors raise: there is no CPU path.
"""
from __future__ import annotations

from math import prod
from typing import Optional

import torch
from torch.nn.modules import module as _nn_module

from . import _lib
from .utils import EasierJitException


def _require_cuda(t: torch.Tensor, what: str) -> None:
    if not (isinstance(t, torch.Tensor) and t.is_cuda):
        raise EasierJitException(f"{what}: easier_gb300 runs on CUDA tensors only (got {getattr(t, 'device', type(t))})")


def select(sel, tensor: torch.Tensor) -> torch.Tensor:
    """Selector.forward: tensor[idx] (easier/core/module.py:364-371)."""
    _require_cuda(tensor, "Selector")
    idx = sel._idx32
    index = tensor.get_device()
    if idx.get_device() != index:
        raise EasierJitException("Selector input is on a different device than its index")
    shape = tensor.shape
    if sel._idx_max >= shape[0]:
        raise IndexError(f"index {sel._idx_max} is out of bounds for dimension 0 with size {shape[0]}")
    src = tensor.contiguous()
    m = idx.shape[0]
    out = torch.empty((m, *shape[1:]), dtype=src.dtype, device=src.device)
    _lib.call("esr_gather", src.data_ptr(), shape[0], src.element_size() * prod(shape[1:]), idx.data_ptr(), m,
              out.data_ptr(), _lib.stream_handle(index))
    return out


def _perm_ptr(red):
    """The Reducer's permutation, or NULL where it is the identity (edges
    already in row order: the kernels then need not read it)."""
    return None if red._in_row_order else _lib.ptr(red._perm32)


def reduce(red, tensor: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Reducer.forward: out.scatter_reduce_(0, idx, t, op, include_self=False)
    (easier/core/module.py:441-461), as a deterministic in-order segment
    reduction over the CSR of idx.  Without ``out`` the kernel writes the
    zeros of unreferenced rows itself."""
    _require_cuda(tensor, "Reducer")
    op = _lib.REDUCE_OPS[red.reduce]
    if out is None:
        out = torch.empty((red.n, *tensor.shape[1:]), dtype=tensor.dtype, device=tensor.device)
        op |= _lib.REDUCE_FILL
    else:
        _require_cuda(out, "Reducer out")
    if tensor.dtype != out.dtype:
        raise RuntimeError(f"scatter_reduce(): Expected self.dtype to be equal to src.dtype ({out.dtype} vs {tensor.dtype})")
    m = red._perm32.shape[0]
    row = tensor.shape[1:]
    if tensor.shape[0] < m or row != out.shape[1:]:
        raise RuntimeError(
            f"Reducer: input of shape {tuple(tensor.shape)} does not match idx length {m} and"
            f" out shape {tuple(out.shape)}")
    src = tensor.contiguous()
    dst = out if out.is_contiguous() else out.contiguous()
    _lib.call("esr_segreduce", _lib.dtype_code(src.dtype), op, src.data_ptr(), prod(row), red._rowptr32.data_ptr(),
              _perm_ptr(red), red.n, dst.data_ptr(), _lib.stream_handle(src.get_device()))
    if dst is not out:
        out.copy_(dst)
    return out


def _plain_call(mod) -> bool:
    """Calling ``mod`` runs its class's forward and nothing else."""
    return "forward" not in mod.__dict__ and not (mod._forward_hooks or mod._forward_pre_hooks or mod._backward_hooks
                                                  or mod._backward_pre_hooks)


def _observed() -> bool:
    """Something watches torch operations (modes, tracing, forward-mode AD,
    vmap, global module hooks): fused paths would hide them."""
    C = torch._C
    return bool(C._len_torch_dispatch_stack() or C._len_torch_function_stack() or C._get_tracing_state() is not None
                or torch.autograd.forward_ad._current_level >= 0 or C._functorch.maybe_current_level() is not None
                or torch.compiler.is_compiling()
                or _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks
                or _nn_module._global_backward_hooks or _nn_module._global_backward_pre_hooks)


def linsys_apply(A, x: torch.Tensor) -> Optional[torch.Tensor]:
    """reducer(selector(x) * Ae) + x * Av in one kernel (esr_linsys_apply,
    bitwise the five-step form), or None where the five steps could do
    anything else: other shapes and dtypes (broadcasts, promotion), gradients,
    hooks, subclasses, an index out of range."""
    sel, red, Ae, Av = A.selector, A.reducer, A.Ae, A.Av
    plain, Selector, Reducer = _linsys_types or _set_linsys_types()
    if (type(sel) is not Selector or type(red) is not Reducer or red.reduce != "sum"
            or sel.easier_index_status != "rewritten" or red.easier_index_status != "rewritten"
            or not _plain_call(sel) or not _plain_call(red) or _observed()):
        return None
    if type(x) not in plain or x.dim() != 1 or not x.is_cuda or x.layout is not torch.strided:
        return None
    dtype, index, grads = x.dtype, x.get_device(), torch.is_grad_enabled()
    if (dtype is not torch.float32 and dtype is not torch.float64) or (grads and x.requires_grad):
        return None
    n, m, col = red.n, red._perm32.shape[0], sel._idx32
    for t, length in ((Ae, m), (Av, n)):
        if (type(t) not in plain or t.dim() != 1 or t.dtype is not dtype or t.get_device() != index
                or (grads and t.requires_grad) or t.shape[0] != length or not t.is_contiguous()):
            return None
    if (x.shape[0] != n or col.shape[0] != m or sel._idx_max >= n or col.get_device() != index
            or red._perm32.get_device() != index):
        return None
    x = x.contiguous()
    y = torch.empty_like(x, requires_grad=False)
    _lib.call("esr_linsys_apply", _lib.dtype_code(dtype), x.data_ptr(), Ae.data_ptr(), Av.data_ptr(), col.data_ptr(),
              red._rowptr32.data_ptr(), _perm_ptr(red), n, y.data_ptr(), _lib.stream_handle(index))
    return y


_linsys_types = None  # (module.py imports this file)


def _set_linsys_types():
    global _linsys_types
    from .module import Reducer, Selector, Tensor
    _linsys_types = ((torch.Tensor, torch.nn.Parameter, Tensor), Selector, Reducer)
    return _linsys_types


_AGG = {"sum": _lib.AGG_SUM, "prod": _lib.AGG_PROD, "norm": _lib.AGG_NORM, "max": _lib.AGG_MAX, "min": _lib.AGG_MIN}


def aggregate(tensor: torch.Tensor, kind: str) -> torch.Tensor:
    """esr.sum/prod/norm/max/min: op over dim 0 with keepdim
    (easier/core/module.py:825-884); FP64 accumulation, fixed order."""
    _require_cuda(tensor, f"esr.{kind}")
    if kind == "norm" and not tensor.dtype.is_floating_point:
        raise RuntimeError("norm(): input dtype should be floating point")
    if kind in ("max", "min") and tensor.shape[0] == 0:
        raise IndexError(f"{kind}(): Expected reduction dim 0 to have non-zero size.")
    src = tensor.contiguous()
    n = src.shape[0]
    cols = prod(src.shape[1:])
    device = src.device
    out = torch.empty((1, *src.shape[1:]), dtype=src.dtype, device=device)
    nbytes = _lib.lib().esr_aggregate_workspace_bytes(n, cols)
    ws = torch.empty(max(int(nbytes), 16), dtype=torch.uint8, device=device)
    _lib.call("esr_aggregate", _lib.dtype_code(src.dtype), _AGG[kind], src.data_ptr(), n, cols, out.data_ptr(),
              ws.data_ptr(), _lib.stream_handle(device))
    return out


def dot(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor = None, workspace: torch.Tensor = None) -> torch.Tensor:
    """FP64-accumulated dot product of two equal-length vectors; returns a
    1-element FP64 device tensor."""
    _require_cuda(a, "dot")
    if a.shape != b.shape or a.dtype != b.dtype:
        raise ValueError("dot: operands must have equal shape and dtype")
    n = a.numel()
    if out is None:
        out = torch.empty(1, dtype=torch.float64, device=a.device)
    if workspace is None:
        workspace = torch.zeros(int(_lib.lib().esr_dot_workspace_bytes(n)), dtype=torch.uint8, device=a.device)
    _lib.call("esr_dot", _lib.dtype_code(a.dtype), _lib.ptr(a.contiguous()), _lib.ptr(b.contiguous()), n,
              _lib.ptr(out), _lib.ptr(workspace), _lib.stream_handle(a.device))
    return out


def device_status(clear: bool = True, device=None) -> int:
    """OR of the device-side error bits raised since the last clear."""
    import ctypes
    v = ctypes.c_int(0)
    _lib.call("esr_device_status", ctypes.byref(v), 1 if clear else 0, _lib.stream_handle(device))
    return v.value
