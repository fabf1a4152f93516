"""``fused_field_read`` on the CUDA library: the drop-in for the reference's operator.

Mirrors ``_ChunkedFieldReadFunction`` / ``fused_field_read`` of the reference
(``field_only_v4_chunked_triton_wiki100.py:912-1123``): same arguments, same
output layout, same gradients, same argument errors. ``block_c`` and ``chunk_t``
are launch hints of the reference's Triton kernels and are accepted and ignored.

``field_read_with_state`` is the same operator with an incoming state and the
outgoing state returned - what the sequence-sharded forward and incremental
decoding need; the reference always starts from the zero state.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def _stream(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


class FieldReadFunction:
    """read, state_out = F(raw, tr, ti, gamma, state_in[, lean]), differentiable (the autograd node
    is native, ``csrc/torch_ops.cpp``).

    With ``lean`` the function does not keep ``read`` for its backward pass but only every
    eighth state row (1/16 of it); the backward kernel recomputes the states in between.
    """

    @staticmethod
    def apply(raw, transition_r, transition_i, gamma, state_in, lean=False):
        return _lib.native().field_read(raw, transition_r, transition_i, gamma, state_in, lean, True)


def fused_field_read_bf16_stats(raw: torch.Tensor, transition_r: torch.Tensor,
                                transition_i: torch.Tensor, gamma: torch.Tensor):
    """``fused_field_read_bf16`` that also returns ``sumsq [B, L]`` (fp32): the sum of squares of
    each token's 4C outputs, which is all an RMS norm over ``read`` needs from it. Both outputs
    are differentiable."""
    return _lib.native().field_read_bf16(raw, transition_r, transition_i, gamma, True)


class MixerEpilogueFunction(torch.autograd.Function):
    """y = x + (acc * rsqrt(sumsq / features + eps) + bias) * sigmoid(gate + gate_bias), one
    kernel each way."""

    @staticmethod
    def forward(ctx, x, acc, gate, sumsq, bias, gate_bias, eps, features):
        lib = _lib.load()
        D = x.shape[-1]
        x, acc, gate = x.contiguous(), acc.contiguous(), gate.contiguous()
        sumsq, bias = sumsq.contiguous().float(), bias.contiguous().float()
        if gate_bias is not None:
            gate_bias = gate_bias.contiguous().float()
        N = x.numel() // D
        y = torch.empty_like(x)
        with torch.cuda.device(x.device):
            rc = lib.fields_mixer_epilogue_forward(_ptr(x), _ptr(acc), _ptr(gate), _ptr(sumsq),
                                                   _ptr(bias), _ptr(gate_bias), _ptr(y), float(eps),
                                                   int(features), N, D, _stream(x.device))
        _lib.check(rc, "fields_mixer_epilogue_forward")
        ctx.save_for_backward(acc, gate, sumsq, bias, gate_bias)
        ctx.consts = (float(eps), int(features), N, D)
        return y

    @staticmethod
    def backward(ctx, grad_y):
        acc, gate, sumsq, bias, gate_bias = ctx.saved_tensors
        eps, features, N, D = ctx.consts
        lib = _lib.load()
        grad_y = grad_y.contiguous().float()
        with torch.cuda.device(grad_y.device):
            grad_acc, grad_gate = torch.empty_like(acc), torch.empty_like(gate)
            grad_sumsq = torch.empty_like(sumsq)
            rows = lib.fields_mixer_epilogue_bias_rows(N)
            bias_rows = torch.empty((2 if gate_bias is not None else 1, rows, D),
                                    device=grad_y.device, dtype=torch.float32)
            rc = lib.fields_mixer_epilogue_backward(
                _ptr(grad_y), _ptr(acc), _ptr(gate), _ptr(sumsq), _ptr(bias), _ptr(gate_bias),
                _ptr(grad_acc), _ptr(grad_gate), _ptr(grad_sumsq), _ptr(bias_rows[0]),
                _ptr(bias_rows[1]) if gate_bias is not None else None, eps, features, N, D,
                _stream(grad_y.device))
            _lib.check(rc, "fields_mixer_epilogue_backward")
            sums = bias_rows.sum(dim=1)
        return (grad_y, grad_acc, grad_gate, grad_sumsq, sums[0],
                sums[1] if gate_bias is not None else None, None, None)


def mixer_epilogue(x: torch.Tensor, acc: torch.Tensor, gate: torch.Tensor, sumsq: torch.Tensor,
                   bias: torch.Tensor, eps: float, features: int,
                   gate_bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x + (acc * rsqrt(sumsq / features + eps) + bias) * sigmoid(gate + gate_bias)`` in one CUDA
    kernel (and one for all gradients): ``x [..., D]`` fp32, ``acc`` and ``gate`` ``[..., D]``
    bfloat16, ``sumsq [...]`` fp32 (per token), ``bias``, ``gate_bias`` ``[D]`` (the latter
    optional); ``D`` a multiple of 4, at most 4096."""
    if x.dtype != torch.float32 or acc.dtype != torch.bfloat16 or gate.dtype != torch.bfloat16:
        raise TypeError((x.dtype, acc.dtype, gate.dtype))
    return MixerEpilogueFunction.apply(x, acc, gate, sumsq, bias, gate_bias, eps, features)


def fused_field_read_bf16(raw: torch.Tensor, transition_r: torch.Tensor,
                          transition_i: torch.Tensor, gamma: torch.Tensor) -> torch.Tensor:
    """The operator on a bfloat16 boundary: ``raw [B, L, 3C]`` bf16 in, ``read [B, L, 4C]`` bf16
    out, fp32 state inside. For mixers that keep the write projection's bf16 output."""
    return _lib.native().field_read_bf16(raw, transition_r, transition_i, gamma, False)


def fused_field_read(raw: torch.Tensor, transition_r: torch.Tensor, transition_i: torch.Tensor,
                     gamma: torch.Tensor, block_c: int = 32, chunk_t: int = 64) -> torch.Tensor:
    """Drop-in for the reference's ``fused_field_read``; returns ``read [B, L, 4C]`` fp32."""
    return _lib.native().field_read(raw, transition_r, transition_i, gamma, None, False, False)


def field_read_with_state(raw, transition_r, transition_i, gamma,
                          state_in: Optional[torch.Tensor] = None, lean: bool = False):
    """Same operator with a carried state: returns ``(read, state_out [B, 2C])``.

    ``lean=True`` keeps only every eighth state row for the backward pass instead of ``read``
    (the kernel recomputes the rest; about 7 % slower backward, 8 KB per token less saved by
    this operator). It pays when the consumer of ``read`` does not keep it either.
    """
    return _lib.native().field_read(raw, transition_r, transition_i, gamma, state_in, lean, True)
