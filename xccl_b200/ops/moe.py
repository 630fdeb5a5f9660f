"""Fused MoE dispatch / combine (``csrc/fused/moe.cu``) on torch tensors."""
from __future__ import annotations

import ctypes as C
from typing import Any, Sequence

import torch

from .. import _capi as K
from ..api import XcclError
from ._args import pointers as _ptrs, stream

_pp = C.POINTER(C.c_void_p)
K.optional("xccl_moe_ws_create", C.c_int, C.POINTER(K.Oob), C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, _pp)
K.optional("xccl_moe_ws_destroy", None, C.c_void_p)
K.optional("xccl_moe_dispatch", C.c_int, C.c_void_p, _pp, _pp, C.c_void_p)
K.optional("xccl_moe_combine", C.c_int, C.c_void_p, _pp, _pp, _pp, C.c_void_p)
K.optional("xccl_moe_ws_buffer", C.c_void_p, C.c_void_p, C.c_int, C.c_int)
K.optional("xccl_moe_ws_cap_rows", C.c_int, C.c_void_p)
K.optional("xccl_moe_ws_error", C.c_uint32, C.c_void_p)

BUF_RECV, BUF_EXPERT_OUT, BUF_EXPERT_ROWS, BUF_ROW_SOURCE = range(4)


class _Workspace:
    """The native workspace; its memory is freed with the last reference to it. One that is still referenced when the
    interpreter ends goes with the process."""

    def __init__(self, h: C.c_void_p):
        self.h = h

    def __del__(self):
        load = getattr(K, "load", None)      # the module may be gone by then
        if load is not None:
            load().xccl_moe_ws_destroy(self.h)


def _view(ptr: int, shape: tuple, dtype: torch.dtype, device, owner: _Workspace) -> torch.Tensor:
    """A tensor on workspace memory. It keeps the workspace: the memory outlives ``MoeWorkspace.close`` for as long as a
    view of it does."""
    n = 1
    for s in shape:
        n *= s
    typestr = {torch.bfloat16: "<i2", torch.int32: "<i4", torch.uint32: "<u4"}[dtype]

    class _Mem:
        __cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}

    mem = _Mem()
    mem.owner = owner          # the tensor's storage holds `mem`
    t = torch.as_tensor(mem, device=device)
    return (t.view(torch.bfloat16) if dtype == torch.bfloat16 else t).view(shape)


class MoeWorkspace:
    """Buffers and state of the fused expert all-to-all for fixed (tokens, hidden, experts, top-k)."""

    def __init__(self, tokens: int, hidden: int, experts: int, topk: int, oob: Any = None, emu_ranks: int = 1,
                 cap_rows: int = 0):
        self.T, self.H, self.E, self.K = tokens, hidden, experts, topk
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.h = C.c_void_p()
        st = K.load().xccl_moe_ws_create(C.byref(oob.c) if oob is not None else None, emu_ranks, tokens, hidden,
                                         experts, topk, cap_rows, C.byref(self.h))
        if st != K.OK:
            raise XcclError(st, "xccl_moe_ws_create")
        self._ws = _Workspace(self.h)
        self.tp = oob.size if oob is not None else emu_ranks
        self.n_local = 1 if oob is not None else emu_ranks
        self.cap_rows = int(K.load().xccl_moe_ws_cap_rows(self.h))

    def _buf(self, local: int, which: int) -> int:
        return int(K.load().xccl_moe_ws_buffer(self.h, local, which))

    def recv(self, local: int = 0) -> torch.Tensor:
        return _view(self._buf(local, BUF_RECV), (self.cap_rows, self.H), torch.bfloat16, self.device, self._ws)

    def expert_out(self, local: int = 0) -> torch.Tensor:
        return _view(self._buf(local, BUF_EXPERT_OUT), (self.cap_rows, self.H), torch.bfloat16, self.device, self._ws)

    def expert_rows(self, local: int = 0) -> torch.Tensor:
        return _view(self._buf(local, BUF_EXPERT_ROWS), (self.E // self.tp + 1,), torch.int32, self.device, self._ws)

    def row_source(self, local: int = 0) -> torch.Tensor:
        return _view(self._buf(local, BUF_ROW_SOURCE), (self.cap_rows,), torch.int32, self.device, self._ws)

    def dispatch(self, x: Sequence[torch.Tensor], ids: Sequence[torch.Tensor]) -> None:
        st = K.load().xccl_moe_dispatch(self.h, _ptrs(x), _ptrs(ids), stream())
        if st != K.OK:
            raise XcclError(st, "xccl_moe_dispatch")

    def combine(self, ids: Sequence[torch.Tensor], weights: Sequence[torch.Tensor], out: Sequence[torch.Tensor]) -> None:
        st = K.load().xccl_moe_combine(self.h, _ptrs(ids), _ptrs(weights), _ptrs(out), stream())
        if st != K.OK:
            raise XcclError(st, "xccl_moe_combine")

    def error(self) -> int:
        torch.cuda.synchronize()
        return int(K.load().xccl_moe_ws_error(self.h))

    def close(self) -> None:
        """Gives the workspace up; its memory is freed now, or with the last tensor that views it. Freeing waits for the
        device, so neither this nor the end of the last view may fall into a graph capture."""
        self.h = C.c_void_p()
        self._ws = None
