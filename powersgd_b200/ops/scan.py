"""Checks and address keys of whole lists of tensors: csrc/host/tensor_scan.cpp where it is built and knows
every object of a list, else the same questions in Python."""
from __future__ import annotations

import importlib.util
import os
from typing import Optional, Sequence

import numpy as np
import torch

from ..csrc.build import SCAN_LIB, scan_target
from ..utils import is_dense, same_layout


def _load(path: str = SCAN_LIB):
    """The extension at `path`; None where there is none or it was compiled for another PyTorch or Python."""
    if not os.path.exists(path):
        return None
    try:
        spec = importlib.util.spec_from_file_location("_tensor_scan", path)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
    except ImportError:   # symbols that are not there
        return None
    return module if getattr(module, "target", None) == scan_target() else None


_native = _load()


def _words(values) -> bytes:
    return np.array(list(values), dtype=np.uint64).tobytes()


def addresses(tensors: Optional[Sequence[Optional[torch.Tensor]]]) -> Optional[bytes]:
    """The addresses of a list, 8 bytes each (0 for None); None for no list."""
    if tensors is None:
        return None
    key = _native.addresses(tensors) if _native is not None else None
    return _words(0 if t is None else t.data_ptr() for t in tensors) if key is None else key


def grad_addresses(params: Sequence[torch.Tensor]) -> bytes:
    """The addresses of the parameters' gradients."""
    key = _native.grad_addresses(params) if _native is not None else None
    return _words(p.grad.data_ptr() for p in params) if key is None else key


def sizes(tensors: Sequence[torch.Tensor]) -> bytes:
    """The numbers of elements of a list, 8 bytes each."""
    key = _native.sizes(tensors) if _native is not None else None
    return _words(t.numel() for t in tensors) if key is None else key


def usable(tensors: Sequence[torch.Tensor], contiguous: bool = False) -> bool:
    """Are all of a list float32 tensors on a GPU, and dense (or contiguous)?"""
    known = _native.usable(tensors, contiguous) if _native is not None else None
    if known is not None:
        return known
    f32 = torch.float32
    return all(t.is_cuda and t.dtype == f32 and (t.is_contiguous() or (not contiguous and is_dense(t))) for t in tensors)


def step_fits(optimizer: torch.optim.Optimizer) -> bool:
    """Does every group, parameter, gradient and momentum buffer of an SGD optimizer suit the fused step? Float32
    dense parameters whose gradients and buffers are laid out like them, momentum buffers for all or none
    of a group."""
    known = _native.step_fits(optimizer.param_groups, optimizer.state) if _native is not None else None
    if known is not None:
        return known
    state, f32 = optimizer.state, torch.float32
    for group in optimizer.param_groups:
        if group.get("maximize", False) or group.get("differentiable", False):
            return False
        buffers = 0
        for p in group["params"]:
            grad = p.grad
            if grad is None or p.dtype != f32 or not (p.is_contiguous() or is_dense(p)) or not same_layout(grad, p):
                return False
            own = state.get(p)
            buf = own.get("momentum_buffer") if own else None
            if buf is not None:
                buffers += 1
                if not same_layout(buf, p):
                    return False
        if buffers and buffers != len(group["params"]):
            return False
    return True
