"""What the plan of the native inference path accepts, and what it notices afterwards (``fields_lm_b200.stack``; no
GPU: a plan only looks at the model)."""
import copy
import pickle

import pytest
import torch
import torch.nn.functional as F

import mirror
from fields_lm_b200 import mixer, stack


class LM(torch.nn.Module):
    def __init__(self, dim=64, layers=2, hidden=32):
        super().__init__()
        self.emb = torch.nn.Embedding(97, dim)
        self.blocks = torch.nn.ModuleList(mirror.FieldBlock(dim, ff_hidden=hidden) for _ in range(layers))
        self.final_norm = mirror.RMSNorm(dim)
        self.lm_head = torch.nn.Linear(dim, 97, bias=False)


def _plan(model):
    return stack.plan(model, torch.device("cpu"))


def _patch(cls, monkeypatch):
    monkeypatch.setattr(cls, "forward", lambda self, x: x)


CHANGES = {
    "eps of a norm": lambda m, mp: setattr(m.blocks[1].ff_norm, "eps", 1e-2),
    "eps of the final norm": lambda m, mp: setattr(m.final_norm, "eps", 1e-2),
    "forward of a norm": lambda m, mp: setattr(m.blocks[0].mixer.read_norm, "forward", lambda x: x),
    "forward of a projection": lambda m, mp: setattr(m.blocks[0].mixer.write_proj, "forward", lambda x: x),
    "forward of the feed-forward": lambda m, mp: setattr(m.blocks[1].ff, "forward", lambda x: x),
    "training mode": lambda m, mp: m.eval(),
    "forward of the norm class": lambda m, mp: _patch(mirror.RMSNorm, mp),
    "forward of the feed-forward class": lambda m, mp: _patch(mirror.PackedSwiGLU, mp),
    "forward of nn.Linear": lambda m, mp: _patch(torch.nn.Linear, mp),
    "attribute of a norm": lambda m, mp: setattr(m.blocks[0].ff_norm, "scale", 2.0),
    "buffer of a norm": lambda m, mp: m.blocks[0].ff_norm.register_buffer("scale", torch.ones(1)),
    "bias of a norm": lambda m, mp: setattr(m.blocks[0].ff_norm, "bias", torch.nn.Parameter(torch.zeros(64))),
    "child of the feed-forward": lambda m, mp: setattr(m.blocks[0].ff, "drop", torch.nn.Dropout(0.5)),
    "parameter": lambda m, mp: setattr(m.blocks[0].ff.w3, "weight", torch.nn.Parameter(torch.zeros(64, 32))),
    "hook": lambda m, mp: m.blocks[0].ff.register_forward_hook(lambda *a: None),
    "block": lambda m, mp: m.blocks.append(mirror.FieldBlock(64, ff_hidden=32)),
}


@pytest.mark.parametrize("change", CHANGES)
def test_plan_notices(change, monkeypatch):
    model = LM()
    plan = _plan(model)
    assert plan is not None and plan.same_model()
    CHANGES[change](model, monkeypatch)
    assert not plan.same_model()


REFUSED = {
    "forward of a norm": lambda m, mp: setattr(m.blocks[0].ff_norm, "forward", lambda x: x),
    "forward of a projection": lambda m, mp: setattr(m.blocks[0].mixer.gate_proj, "forward", lambda x: x),
    "forward of nn.Linear": lambda m, mp: _patch(torch.nn.Linear, mp),
    "bias of a norm": lambda m, mp: setattr(m.blocks[0].ff_norm, "bias", torch.nn.Parameter(torch.zeros(64))),
    "buffer of a norm": lambda m, mp: m.final_norm.register_buffer("scale", torch.ones(1)),
    "attribute that may change inside": lambda m, mp: setattr(m.blocks[0].ff, "options", {"limit": None}),
    "child of the feed-forward": lambda m, mp: setattr(m.blocks[0].ff, "drop", torch.nn.Dropout(0.0)),
}


@pytest.mark.parametrize("change", REFUSED)
def test_plan_refuses(change, monkeypatch):
    model = LM()
    REFUSED[change](model, monkeypatch)
    assert _plan(model) is None


def test_mixer_leaves_other_forwards_alone(monkeypatch):
    """A write projection whose call is more than F.linear is called by the mixer, not read."""
    m = mirror.IndependentVacancyField(64)
    reached = []
    native = type("Native", (), {"fused_mixer": staticmethod(lambda *a: reached.append(1))})
    monkeypatch.setattr(mixer._lib, "native", lambda: native)
    x = torch.zeros(1, 2, 64)
    mixer._native_mixer(m, x)
    assert len(reached) == 1
    m.write_proj.forward = lambda x: F.linear(x, m.write_proj.weight, m.write_proj.bias)
    mixer._native_mixer(m, x)
    del m.write_proj.forward
    hook = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        mixer._native_mixer(m, x)
    finally:
        hook.remove()
    assert len(reached) == 1
    mixer._native_mixer(m, x)
    assert len(reached) == 2


def test_comparison_does_not_rest_on_the_weights():
    """A feed-forward of another formula is found out although its weights are zero, and one refusal is enough."""
    class PackedSwiGLU(mirror.PackedSwiGLU):
        def forward(self, x):
            gate, value = self.w12(x).chunk(2, dim=-1)
            return self.w3(F.gelu(gate) * value)

    model = LM()
    for block in model.blocks:
        block.ff.__class__ = PackedSwiGLU
        torch.nn.init.zeros_(block.ff.w3.weight)
    plan = _plan(model)
    assert not plan.usable and plan.same_model()
    odd = LM()
    odd.blocks[1].ff.__class__ = PackedSwiGLU  # one of several
    assert not _plan(odd).usable
    for m in (LM(), LM().requires_grad_(False)):
        torch.nn.init.constant_(m.blocks[0].ff.w3.weight, float("nan"))  # to be loaded yet
        assert _plan(m).usable


def test_decoder_keeps_plan_and_refusal(monkeypatch):
    from fields_lm_b200 import FieldStackDecoder
    made = []
    plan = stack.plan
    monkeypatch.setattr(stack, "plan", lambda *a: made.append(1) or plan(*a))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    x = torch.zeros(1, 64)
    model = LM()
    dec = FieldStackDecoder(model)
    first = dec._native_stack(x)
    dec.reset()
    assert first is not None and dec._native_stack(x) is first and made == [1]
    model.blocks[0].ff_norm.eps = 1e-3
    assert dec._native_stack(x) not in (None, first) and made == [1, 1]
    mirror_forward = mirror.PackedSwiGLU.forward
    monkeypatch.setattr(mirror.PackedSwiGLU, "forward", lambda self, x: 2 * mirror_forward(self, x))
    assert dec._native_stack(x) is None and dec._native_stack(x) is None and made == [1, 1, 1] and dec._refused
    monkeypatch.undo()
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    assert dec._native_stack(x) is not None and not dec._refused


def test_comparison_leaves_the_model_alone():
    class PackedSwiGLU(mirror.PackedSwiGLU):
        def forward(self, x):
            assert self is not model.blocks[0].ff
            return super().forward(x[:, None])  # a formula that fails is a refusal

    model = LM()
    before = {k: (v, v.clone()) for k, v in model.state_dict(keep_vars=True).items()}
    model.blocks[0].ff.__class__ = PackedSwiGLU
    assert _plan(model) is None or not _plan(model).usable
    for k, v in model.state_dict(keep_vars=True).items():
        assert v is before[k][0] and torch.equal(v, before[k][1])


def test_decoder_can_be_copied_and_pickled(monkeypatch):
    from fields_lm_b200 import FieldStackDecoder
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    dec = FieldStackDecoder(LM())
    dec.states = [torch.ones(1, 64), torch.ones(1, 64)]
    plan = dec._native_stack(torch.zeros(1, 64))
    for twin in (copy.copy(dec), copy.deepcopy(dec), pickle.loads(pickle.dumps(dec))):
        assert twin._stack is None and torch.equal(twin.states[1], dec.states[1])
        assert twin._native_stack(torch.zeros(1, 64)) is not None
    assert dec._stack is plan
