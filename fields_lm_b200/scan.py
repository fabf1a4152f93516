"""``hierarchical_scan`` for real fp32 CUDA tensors on the CUDA library.

The reference's scan primitive ``hierarchical_scan(a, b, block=32)``
(``field_only_v4_chunked_triton_wiki100.py:347-391``) has a second call site besides the
Field read: the softpatch ``FastBoundaryStateMixer`` runs it on a rank-64 real state with one
decay per token expanded over the channels
(``official_source/field_hybrid_speed_optimization_v6.py:333-335``). ``linear_scan`` is that
call on this library's ``fields_scan_forward`` / ``fields_scan_backward``: same arguments, same
output ``[B, L, C]``, gradients for ``a`` and ``b``, the same ``ValueError`` for ``block``
outside ``[1, 64]`` (``block`` itself is a blocking hint of the reference and does not change
the result).

``scan_entry(original)`` builds the function that :func:`fields_lm_b200.install` puts in place
of the module global: real fp32 CUDA inputs run here, everything else (the complex CPU call of
``reference_field_read``) goes to the reference's own function untouched.
"""
from __future__ import annotations

from typing import Callable, Optional

import torch

from . import _lib


def linear_scan(a: torch.Tensor, b: torch.Tensor, block: int = 32) -> torch.Tensor:
    """The reference's ``hierarchical_scan(a, b, block)`` for real fp32 CUDA tensors."""
    if block < 1 or block > 64:
        raise ValueError("field_chunk must be in [1, 64]")
    return _lib.native().linear_scan(a, b, None, False)


def linear_scan_with_state(a: torch.Tensor, b: torch.Tensor,
                           state_in: Optional[torch.Tensor] = None):
    """The same scan from an incoming state ``[B, C]``; returns (states, state after the last
    step). An extension: the reference always starts from zero."""
    return _lib.native().linear_scan(a, b, state_in, True)


def scan_entry(original: Callable) -> Callable:
    """The replacement for a module's ``hierarchical_scan`` global: real fp32 CUDA calls run on
    this library, every other call (complex tensors, CPU tensors, other dtypes) goes to
    ``original`` exactly as before."""

    def hierarchical_scan(a, b, block: int = 32):
        if (torch.is_tensor(a) and torch.is_tensor(b) and a.is_cuda and b.is_cuda
                and a.dtype == torch.float32 and b.dtype == torch.float32
                and a.dim() == 3 and a.shape == b.shape):
            return linear_scan(a, b, block)
        return original(a, b, block)

    hierarchical_scan.__wrapped__ = original
    return hierarchical_scan
