"""Incremental decoding: one recurrent step of the Field read per new token.

The reference has no incremental path (its inference is a full-sequence pass); the
recurrence is causal, so a prefix pass that returns its end state followed by
single-token steps reproduces the full pass over prefix + tokens, which is how the tests
check it. The state ``[B, 2C]`` stays fp32; inputs and outputs are fp32 or bf16.
"""
from __future__ import annotations

import torch

from . import _lib


def field_read_step(raw_row: torch.Tensor, transition_r: torch.Tensor, transition_i: torch.Tensor,
                    gamma: torch.Tensor, state: torch.Tensor) -> torch.Tensor:
    """Advances ``state`` in place by one token and returns that token's ``read`` row.

    ``raw_row`` is ``[B, 3C]`` (fp32 or bf16, CUDA, contiguous); ``state`` is ``[B, 2C]`` fp32
    and is overwritten with the new state; the result is ``[B, 4C]`` in ``raw_row``'s dtype.
    """
    return _lib.native().step(raw_row, transition_r, transition_i, gamma, state)


class FieldStackDecoder:
    """Stateful prefill -> decode for a language model made of the reference's Field blocks.

    Works on any module shaped like the reference's field-only ``ByteLM``
    (``field_only_v4_chunked_triton_wiki100.py:1306-1344`` with ``model="field_triton"``): an
    embedding ``emb``, a list ``blocks`` of ``FieldBlock``s, ``final_norm`` and ``lm_head``. The
    reference itself can only run the whole sequence again for every new token; here
    :meth:`prefill` runs the prompt once and keeps one fp32 state ``[B, dim]`` per block, and
    :meth:`step` advances all of them by one token. The hybrid ``FieldsForCausalLM`` is not
    covered: its refresh-attention and Mamba-2 layers would need caches of their own.
    """

    def __init__(self, model: torch.nn.Module):
        for name in ("emb", "blocks", "final_norm", "lm_head"):
            if not hasattr(model, name):
                raise TypeError(f"model has no `{name}`: not a field-only language model")
        for block in model.blocks:
            if type(block).__name__ != "FieldBlock":
                raise TypeError(f"block of type {type(block).__name__}: only FieldBlock can be "
                                "stepped")
        self.model = model
        self.states = None
        self._stack = None     # native runner of the blocks (csrc/torch_stack.cpp), where it applies
        self._refused = False  # it did not apply when last asked for (asked again at a prefill)

    def __getstate__(self) -> dict:
        # a copy or an unpickled decoder makes a plan of its own
        return dict(vars(self), _stack=None, _refused=False)

    def reset(self) -> None:
        self.states = None  # (the plan stays: it notices by itself when the model changes)

    @staticmethod
    def _bf16_products(x: torch.Tensor) -> bool:
        """Whether the caller's context is the one the native runner computes: fp32 activations
        under bfloat16 autocast."""
        return (x.is_cuda and x.dtype == torch.float32 and x.numel() > 0
                and torch.is_autocast_enabled("cuda")
                and torch.get_autocast_dtype("cuda") == torch.bfloat16)

    def _native_stack(self, x: torch.Tensor):
        """The runner for the model as it is now, or None; one of its own for a graph that is being
        captured, whose replays have to follow the weights and must not depend on this object."""
        if torch.cuda.is_current_stream_capturing():
            usable = self._stack is not None and self._stack.usable and self._stack.same_model()
            return self._stack.fresh() if usable else None  # (a plan cannot be made here)
        if self._stack is None or not self._stack.same_model():
            from .stack import plan
            self._stack = plan(self.model, x.device)
            self._refused = self._stack is None or not self._stack.usable
        return None if self._refused else self._stack

    @torch.no_grad()
    def prefill(self, tokens: torch.Tensor, last_only: bool = True) -> torch.Tensor:
        """Runs the prompt ``tokens [B, T]`` and stores the blocks' end states. Returns the
        logits of the last position ``[B, V]``, or of every position with ``last_only=False``.

        Under bfloat16 autocast the blocks run natively where they are what that path computes
        (``fields_lm_b200.stack``); the weights are laid out for it here, and the steps that
        follow use the same copies until a parameter changes: an in-place write as torch counts
        it (``load_state_dict``, an optimizer, ``copy_`` under ``no_grad``) or another tensor in
        its place. A write that torch does not count, through ``.data`` or into the memory by
        other means, is seen by the next prefill; of what only the steps read (biases, and weights in an
        order of theirs, which the first step lays out) by a step as well. Inference tensors, which
        have no count, are laid out for every step."""
        from .mixer import block_prefill
        x = self.model.emb(tokens)
        if self._bf16_products(x) and x.dim() == 3:
            stack = self._native_stack(x)
            if stack is not None:
                stack.layout(x.shape[0] * x.shape[1], x.shape[0])
                x, self.states = stack.prefill(x)
                return self.model.lm_head(self.model.final_norm(x[:, -1] if last_only else x))
        states = []
        for block in self.model.blocks:
            x, state = block_prefill(block, x)
            states.append(state)
        self.states = states
        if last_only:
            x = x[:, -1]
        return self.model.lm_head(self.model.final_norm(x))

    @torch.no_grad()
    def step(self, tokens: torch.Tensor) -> torch.Tensor:
        """One new token per sequence, ``tokens [B]``; returns its logits ``[B, V]``."""
        from .mixer import block_step
        if self.states is None:
            raise RuntimeError("call prefill() before step()")
        x = self.model.emb(tokens)
        if not self._refused and self._bf16_products(x) and x.dim() == 2:
            stack = self._stack
            if (stack is None or not stack.current()  # something has changed since the prefill
                    or torch.cuda.is_current_stream_capturing()):
                stack = self._native_stack(x)
                if stack is not None:
                    stack.layout(0, x.shape[0])
            if stack is not None:
                out = stack.step(x, self.states)
                return out if stack.has_head else self.model.lm_head(self.model.final_norm(out))
        for block, state in zip(self.model.blocks, self.states):
            x = block_step(block, x, state)
        return self.model.lm_head(self.model.final_norm(x))

    @torch.no_grad()
    def generate(self, prompt: torch.Tensor, new_tokens: int) -> torch.Tensor:
        """Greedy continuation of ``prompt [B, T]`` by ``new_tokens`` tokens."""
        logits = self.prefill(prompt)
        out = [prompt]
        for _ in range(new_tokens):
            nxt = logits.argmax(dim=-1)
            out.append(nxt[:, None])
            logits = self.step(nxt)
        return torch.cat(out, dim=1)
