"""Recognises a stack of the reference's Field blocks that the native inference path can run.

``plan(model, device)`` looks at a field-only language model (the reference's ``ByteLM``,
``field_only_v4_chunked_triton_wiki100.py:1306-1344``) and returns a ``FieldStack``
(``csrc/torch_stack.cpp``) that runs its blocks under bfloat16 autocast with a handful of launches
per block, or None if any part of the model is not what that path computes: other module
classes, hooks, parameters that are not dense fp32 tensors on one GPU, sizes the kernels do not
take. The feed-forward and the norms are modules of the model's own, so each kind of them is also
run once, on a small input and weights made for it, and compared with the formula the kernels use
(the model's own weights could hide a difference: zeros do). What that comparison rests on is part of
the plan: the class's ``forward`` and the instance's attributes, which therefore have to be plain
values, beside the parameters, children and hooks. A kind is a class, a size and attributes: 18 blocks
have four of them and 55 modules, whose comparisons took 9 ms of the first prefill.
"""
from __future__ import annotations

import copy
import types
from typing import List, Optional

import torch
import torch.nn.functional as F

from . import _lib
from .mixer import plain_linear

_HOOKS = ("_forward_hooks", "_forward_pre_hooks")
_OWN = frozenset(vars(torch.nn.Module()))  # what every module's __dict__ holds
_PLAIN = (int, float, bool, str, type(None), torch.dtype, types.FunctionType, types.BuiltinFunctionType)


class _NotApplicable(Exception):
    pass


def _need(ok: bool) -> None:
    if not ok:
        raise _NotApplicable


def _twin(module: torch.nn.Module, weights: dict, prefix: str = "") -> torch.nn.Module:
    """A copy of ``module`` around other weights; the module itself may be in use by another thread."""
    twin = copy.copy(module)
    vars(twin)["_parameters"] = {k: p if p is None else weights[prefix + k] for k, p in module._parameters.items()}
    vars(twin)["_modules"] = {k: m and _twin(m, weights, prefix + k + ".") for k, m in module._modules.items()}
    return twin


class _Survey:
    """Collects what the plan depends on: parameters, the slots they sit in, dictionaries and their
    sizes (hooks: none), classes and their ``forward``, and how far each module is from the formula it
    is taken for."""

    def __init__(self, device):
        self.device = device
        self.slots, self.sizes = [], []
        self.classes, self.errors = {}, {}

    def child(self, module, name: str):
        _need(name in module._modules)
        child = module._modules[name]
        self.slots.append((module._modules, name, child))
        self.no_hooks(*(getattr(child, h) for h in _HOOKS))
        _need("forward" not in vars(child))  # (nor later: the size of the dictionary is kept)
        self.sizes.append((vars(child), len(vars(child))))
        return child

    def no_hooks(self, *dicts) -> None:
        _need(not any(dicts))
        self.sizes += [(d, 0) for d in dicts]

    def formula(self, module, parameters: set, children: set) -> None:
        """A module that is taken for a formula: nothing in it beside these but plain attributes."""
        for own, names in ((module._parameters, parameters), (module._modules, children), (module._buffers, set())):
            _need({k for k, v in own.items() if v is not None} == names)
            self.slots += [(own, k, None) for k, v in own.items() if v is None]
            self.sizes.append((own, len(own)))
        for key, value in vars(module).items():
            if key not in _OWN:
                items = value if type(value) is tuple else (value,)
                _need(all(isinstance(v, _PLAIN) for v in items))
            if key not in _OWN or key == "training":
                self.slots.append((vars(module), key, value))
        self.classes[type(module)] = type(module).forward

    def parameter(self, module, name: str, *shape: int) -> torch.Tensor:
        _need(name in module._parameters)
        p = module._parameters[name]
        _need(isinstance(p, torch.Tensor) and p.dtype == torch.float32 and p.device == self.device
              and tuple(p.shape) == shape and p.is_contiguous() and p.data_ptr() % 16 == 0)
        self.slots.append((module._parameters, name, p))
        return p

    def linear(self, module, name: str, rows: int, cols: int, bias: bool):
        lin = self.child(module, name)
        _need(plain_linear(lin) and (lin.bias is not None) == bias)
        self.classes[torch.nn.Linear] = torch.nn.Linear.forward
        weight = self.parameter(lin, "weight", rows, cols)
        return (weight, self.parameter(lin, "bias", rows)) if bias else (weight, None)

    def norm(self, module, name: str, dim: int):
        norm = self.child(module, name)
        _need(type(norm).__name__ == "RMSNorm" and isinstance(getattr(norm, "eps", None), float))
        weight = self.parameter(norm, "weight", dim)
        self.formula(norm, {"weight"}, set())
        self.compare(norm, dim, lambda x, w: x * torch.rsqrt(x.square().mean(-1, keepdim=True) + norm.eps) * w["weight"])
        return weight, norm.eps

    def compare(self, module, dim: int, formula) -> None:
        shapes = tuple((name, tuple(p.shape)) for name, p in module.named_parameters())
        kind = (type(module), dim, shapes, module.training,
                tuple(sorted((k, v) for k, v in vars(module).items() if k not in _OWN)))
        if kind in self.errors:
            return

        gen = torch.Generator(self.device).manual_seed(0)
        x = torch.randn(2, dim, device=self.device, generator=gen)
        weights = {name: torch.randn(shape, device=self.device, generator=gen) / (shape[-1] ** 0.5 if len(shape) > 1 else 1)
                   for name, shape in shapes}
        want = formula(x, weights)
        try:
            got = _twin(module, weights)(x)
        except Exception:
            raise _NotApplicable
        _need(got.shape == want.shape and got.dtype == want.dtype)
        self.errors[kind] = (got - want).abs().max() / want.abs().max().clamp_min(1e-6)


def _block(s: _Survey, blocks, key: str, dim: int):
    block = s.child(blocks, key)
    _need(type(block).__name__ == "FieldBlock")
    mixer = s.child(block, "mixer")
    _need(type(mixer).__name__ == "IndependentVacancyField" and mixer.dim == dim
          and 2 * mixer.channels == dim)
    channels = dim // 2
    write = s.linear(mixer, "write_proj", 3 * channels, dim, True)
    gate = s.linear(mixer, "gate_proj", dim, dim, True)
    out = s.linear(mixer, "out_proj", dim, 2 * dim, True)
    read_norm, read_eps = s.norm(mixer, "read_norm", 2 * dim)
    ff_norm, ff_eps = s.norm(block, "ff_norm", dim)
    ff = s.child(block, "ff")
    _need(type(ff).__name__ == "PackedSwiGLU" and "w3" in ff._modules)
    hidden = ff._modules["w3"].weight.shape[1]
    _need(hidden % 8 == 0)
    w12, _ = s.linear(ff, "w12", 2 * hidden, dim, False)
    w3, _ = s.linear(ff, "w3", dim, hidden, False)

    def feed_forward(x, w):
        u, v = F.linear(x, w["w12.weight"]).chunk(2, dim=-1)
        return F.linear(F.silu(u) * v, w["w3.weight"])

    s.formula(ff, set(), {"w12", "w3"})
    s.compare(ff, dim, feed_forward)
    radius = s.parameter(mixer, "radius_logit", channels)
    theta = s.parameter(mixer, "theta", channels)
    return [*write, *gate, *out, read_norm, ff_norm, w12, w3, radius, theta], (read_eps, ff_eps), hidden


@torch.no_grad()
def plan(model: torch.nn.Module, device: torch.device) -> Optional[object]:
    """The native runner for ``model``'s blocks, or None if they are not what it computes. One that
    is not ``usable`` stands for a model that only the comparison refused, so that it need not be
    repeated. Reads a value back, so not while a graph is being captured."""
    s = _Survey(device)
    try:
        with torch.autocast("cuda", enabled=False):
            s.no_hooks(*(getattr(torch.nn.modules.module, "_global" + h) for h in _HOOKS))
            blocks = s.child(model, "blocks")
            _need(len(blocks) > 0 and type(blocks) is torch.nn.ModuleList)
            first = blocks[0]
            dim = int(getattr(getattr(first, "mixer", None), "dim", 0))
            _need(dim > 0 and dim % 8 == 0 and dim <= 4096)
            params: List[list] = []
            eps, widths = [], set()
            for key in blocks._modules:
                p, e, hidden = _block(s, blocks, key, dim)
                params.append(p)
                eps.append(e)
                widths.add(hidden)
            _need(len(widths) == 1)
            tail, tail_eps = [], 0.0
            head = model._modules.get("lm_head")
            if isinstance(head, torch.nn.Linear) and plain_linear(head) and not any(getattr(head, h) for h in _HOOKS):
                weight, tail_eps = s.norm(model, "final_norm", dim)
                w, b = s.linear(model, "lm_head", head.weight.shape[0], dim, head.bias is not None)
                tail = [weight, w] + ([] if b is None else [b])
            usable = float(torch.stack(list(s.errors.values())).max()) < 1e-4
    except (_NotApplicable, AttributeError):
        return None
    sizes = s.sizes + [(blocks._modules, len(params))]
    return _lib.native().FieldStack(params, eps, s.slots, sizes, list(s.classes.items()), tail, tail_eps, usable)
