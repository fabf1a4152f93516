"""Performance cases: the work a user of this package has it do, through its public entry points.

Kinds (key ``kind`` of a case):

* ``operator``  - the Field read, ``fused_field_read`` and its variants, forward and (``grad``)
  backward through autograd. ``form``: ``fp32`` (the drop-in of the training recipe), ``bf16`` (the
  bfloat16 boundary), ``state`` / ``lean`` (``field_read_with_state`` with a state carried in
  and out, without and with the reduced saved activations);
* ``step``      - ``field_read_step``, one recurrent step of incremental decoding;
* ``scan``      - ``linear_scan``, the softpatch mixer's real-valued scan, forward and backward;
* ``mixer``     - ``fused_mixer_forward`` on a Field mixer under bfloat16 autocast, forward and backward
  (what ``install(model, fused_mixer=True)`` runs);
* ``prefill`` / ``decode`` - ``FieldStackDecoder`` on a stack of Field blocks under bfloat16 autocast.

Sizes are the package's own: d_model 1,024 (512 channels), 8 x 2,048 tokens for training, 65,536 for long
context, batch 256 and 18 blocks for decoding, and smaller, odd and ragged ones around them.
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

import fields_lm_b200
from fields_lm_b200 import mixer as field_mixer

VOCAB = 256  # byte-level language model
FF = {1024: 2528, 512: 1344, 256: 704, 128: 352}  # SwiGLU width of a block of that d_model


def listed():
    return [
        # one new token of one sequence through one recurrence: pure call latency
        dict(name="step_1", kind="step", dtype="fp32", B=1, C=512),
        # one new token of a full serving batch through one recurrence
        dict(name="step_256", kind="step", dtype="bf16", B=256, C=512),
        # a short sequence: debugging, evaluation of single prompts; latency of both directions
        dict(name="operator_1x256", kind="operator", form="fp32", grad=True, B=1, L=256, C=512),
        # the operator of the training recipe
        dict(name="operator_8x2048", kind="operator", form="fp32", grad=True, B=8, L=2048, C=512),
        # the same on the bfloat16 boundary
        dict(name="operator_bf16_8x2048", kind="operator", form="bf16", grad=True, B=8, L=2048, C=512),
        # long-context evaluation: forward only, one sequence
        dict(name="operator_fwd_1x65536", kind="operator", form="fp32", grad=False, B=1, L=65536, C=512),
        # a ragged batch of a narrow model whose width does not allow wide accesses
        dict(name="operator_odd_3x777", kind="operator", form="fp32", grad=True, B=3, L=777, C=333),
        # truncated back-propagation: spans that hand their state over, reduced saved activations
        dict(name="operator_lean_2x3001", kind="operator", form="lean", grad=True, B=2, L=3001, C=384),
        # the softpatch mixer's scan of the training recipe: one decay per token, rank-64 state
        dict(name="scan_8x2048x64", kind="scan", shared=True, B=8, L=2048, C=64),
        # training step of one fused Field mixer
        dict(name="mixer_8x2048", kind="mixer", B=8, L=2048, dim=1024),
        # a batch of prompts through the whole stack
        dict(name="prefill_8x1024", kind="prefill", B=8, L=1024, dim=1024, blocks=18),
        # one new token of a full serving batch through the whole stack
        dict(name="decode_256", kind="decode", B=256, L=32, dim=1024, blocks=18),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operator"] * 6 + ["step"] * 2 + ["scan", "mixer", "prefill", "decode"])
    if kind == "operator":
        form = rng.choice(["fp32", "fp32", "fp32", "bf16", "bf16", "state", "lean"])
        # the default width half of the time, any other width otherwise
        C = 512 if rng.random() < 0.5 else _log_uniform(rng, 24, 1024)
        if form != "fp32" or rng.random() < 0.7:
            C -= C % 4  # only the fp32 form takes every channel count
        grad = rng.random() < 0.75
        tokens = _log_uniform(rng, 64, 16384 if grad else 65536)
        B = min(_log_uniform(rng, 1, 16), max(1, tokens // 16))
        # (wide and long together stay within the largest listed sizes)
        L = max(1, min(tokens // B, 16384 * 512 // (B * C) if grad else 65536 * 512 // (B * C)))
        return dict(kind=kind, form=form, grad=grad, B=B, L=L, C=C)
    if kind == "step":
        C = 512 if rng.random() < 0.5 else 4 * _log_uniform(rng, 8, 256)
        return dict(kind=kind, dtype=rng.choice(["fp32", "bf16"]), B=_log_uniform(rng, 1, 512), C=C)
    if kind == "scan":
        B = _log_uniform(rng, 1, 8)
        return dict(kind=kind, shared=rng.random() < 0.7, B=B, L=_log_uniform(rng, 64, 16384 // B),
                    C=rng.choice([64, 64, 32, 100, 128]))
    dim = rng.choice([256, 512, 1024])
    if kind == "mixer":
        B = _log_uniform(rng, 1, 8)
        return dict(kind=kind, B=B, L=_log_uniform(rng, 64, 16384 // B), dim=dim)
    blocks = rng.choice([4, 8, 18])
    if kind == "prefill":
        B = _log_uniform(rng, 1, 8)
        return dict(kind=kind, B=B, L=_log_uniform(rng, 16, 8192 // B), dim=dim, blocks=blocks)
    return dict(kind=kind, B=_log_uniform(rng, 1, 256), L=rng.randint(4, 48), dim=dim, blocks=blocks)


# ---------------------------------------------------------------------------------------------
# The modules a user's model consists of: a Field mixer, a Field block and a field-only language
# model, with the attributes the package works on.
# ---------------------------------------------------------------------------------------------
class RMSNorm(nn.Module):
    def __init__(self, dim, eps=1e-6):
        super().__init__()
        self.weight = nn.Parameter(1.0 + 0.1 * torch.randn(dim))
        self.eps = eps

    def forward(self, x):
        xf = x.float()
        inv = torch.rsqrt(xf.pow(2).mean(dim=-1, keepdim=True) + self.eps)
        return (xf * inv * self.weight.float()).to(x.dtype)


class PackedSwiGLU(nn.Module):
    def __init__(self, dim, hidden):
        super().__init__()
        self.hidden = hidden
        self.w12 = nn.Linear(dim, 2 * hidden, bias=False)
        self.w3 = nn.Linear(hidden, dim, bias=False)

    def forward(self, x):
        gate, value = self.w12(x).chunk(2, dim=-1)
        return self.w3(F.silu(gate) * value)


class IndependentVacancyField(nn.Module):
    def __init__(self, dim):
        super().__init__()
        self.dim, self.channels = dim, dim // 2
        self.write_proj = nn.Linear(dim, dim + self.channels)
        ring = torch.linspace(0.85, 0.999, self.channels)
        self.radius_logit = nn.Parameter(torch.log(ring / (1.0 - ring)) + 0.1 * torch.randn(self.channels))
        self.theta = nn.Parameter(torch.linspace(0.03, math.pi * 0.97, self.channels))
        self.read_norm = RMSNorm(2 * dim)
        self.out_proj = nn.Linear(2 * dim, dim)
        self.gate_proj = nn.Linear(dim, dim)


class FieldBlock(nn.Module):
    def __init__(self, dim):
        super().__init__()
        self.mixer = IndependentVacancyField(dim)
        self.ff_norm = RMSNorm(dim)
        self.ff = PackedSwiGLU(dim, FF[dim])


class ByteLM(nn.Module):
    def __init__(self, dim, blocks):
        super().__init__()
        self.emb = nn.Embedding(VOCAB, dim)
        self.blocks = nn.ModuleList(FieldBlock(dim) for _ in range(blocks))
        self.final_norm = RMSNorm(dim)
        self.lm_head = nn.Linear(dim, VOCAB, bias=False)


def _transition(C, gen):
    """lambda = r e^{i theta} and gamma over the ring of radii a mixer starts from, jittered."""
    ring = torch.linspace(0.85, 0.999, C, device="cuda")
    logit = torch.log(ring / (1.0 - ring)) + 0.1 * torch.randn(C, device="cuda", generator=gen)
    theta = torch.linspace(0.03, math.pi * 0.97, C, device="cuda")
    radius = torch.sigmoid(logit).clamp(0.50, 0.99995)
    return [radius * torch.cos(theta), radius * torch.sin(theta),
            torch.sqrt((1.0 - radius.square()).clamp_min(1e-4))]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0):
        return torch.randn(*shape, device="cuda", generator=gen).mul_(scale)

    kind = case["kind"]
    if kind == "operator":
        B, L, C = case["B"], case["L"], case["C"]
        bf16 = case["form"] == "bf16"
        # the scale a write projection gives at initialisation
        raw = normal(B, L, 3 * C, scale=0.577)
        s = dict(case=case, leaves=[raw.bfloat16() if bf16 else raw, *_transition(C, gen)])
        if case["form"] in ("state", "lean"):
            s["leaves"].append(normal(B, 2 * C, scale=0.3))
        if case["grad"]:
            for t in s["leaves"]:
                t.requires_grad_(True)
            grad = normal(B, L, 4 * C)
            s["grads"] = [grad.bfloat16() if bf16 else grad]
            if case["form"] in ("state", "lean"):
                s["grads"].append(normal(B, 2 * C))
        return s
    if kind == "step":
        B, C = case["B"], case["C"]
        dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        return dict(case=case, raw=normal(B, 3 * C, scale=0.577).to(dtype), par=_transition(C, gen),
                    state=normal(B, 2 * C, scale=0.3))
    if kind == "scan":
        B, L, C = case["B"], case["L"], case["C"]
        decay = torch.sigmoid(normal(B, L, 1 if case["shared"] else C, scale=1.5)).requires_grad_(True)
        return dict(case=case, a=decay, b=normal(B, L, C).requires_grad_(True), grad=normal(B, L, C))
    torch.manual_seed(seed)
    if kind == "mixer":
        with torch.device("cuda"):
            m = IndependentVacancyField(case["dim"])
        x = normal(case["B"], case["L"], case["dim"]).requires_grad_(True)
        return dict(case=case, mixer=m, x=x, grad=normal(case["B"], case["L"], case["dim"]))
    with torch.device("cuda"):
        model = ByteLM(case["dim"], case["blocks"])
    decoder = fields_lm_b200.FieldStackDecoder(model)
    tokens = torch.randint(0, VOCAB, (case["B"], case["L"]), device="cuda", generator=gen)
    s = dict(case=case, decoder=decoder, tokens=tokens)
    if kind == "decode":
        s["next"] = torch.randint(0, VOCAB, (case["B"],), device="cuda", generator=gen)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            decoder.prefill(tokens)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "operator":
        form, leaves = case["form"], s["leaves"]

        def forward():
            if form == "fp32":
                return (fields_lm_b200.fused_field_read(*leaves),)
            if form == "bf16":
                return (fields_lm_b200.fused_field_read_bf16(*leaves),)
            return fields_lm_b200.field_read_with_state(*leaves, lean=form == "lean")

        if not case["grad"]:
            with torch.no_grad():
                return forward()
        out = forward()
        return out + torch.autograd.grad(out, leaves, s["grads"])
    if kind == "step":
        return fields_lm_b200.field_read_step(s["raw"], *s["par"], s["state"]), s["state"]
    if kind == "scan":
        a = s["a"].expand_as(s["b"])
        states = fields_lm_b200.linear_scan(a, s["b"])
        return (states,) + torch.autograd.grad(states, [s["a"], s["b"]], s["grad"])
    with torch.autocast("cuda", dtype=torch.bfloat16):
        if kind == "mixer":
            y = field_mixer.fused_mixer_forward(s["mixer"], s["x"])
        elif kind == "prefill":
            return (s["decoder"].prefill(s["tokens"]), *s["decoder"].states)
        else:
            return (s["decoder"].step(s["next"]), *s["decoder"].states)
    return (y,) + torch.autograd.grad(y, [s["x"], *s["mixer"].parameters()], s["grad"])


def work(case):
    kind, B = case["kind"], case["B"]
    if kind == "operator":
        n = B * case["L"] * case["C"]
        size = 2 if case["form"] == "bf16" else 4
        # raw in, read out; with a backward pass grad_read in and grad_raw out as well
        return {"bytes": n * size * (14 if case["grad"] else 7), "flops": n * (110 if case["grad"] else 35)}
    if kind == "step":
        n = B * case["C"]
        return {"bytes": n * (16 + 7 * (2 if case["dtype"] == "bf16" else 4)), "flops": n * 35}
    if kind == "scan":
        n, decays = B * case["L"] * case["C"], B * case["L"] * (1 if case["shared"] else case["C"])
        # drive and decay in, states out, their gradient in, two gradients out
        return {"bytes": 4 * (4 * n + 2 * decays), "flops": 7 * n}
    dim = case["dim"]
    mixer_weights = dim * (3 * dim // 2) + 2 * dim * dim + dim * dim
    if kind == "mixer":
        n = B * case["L"]
        # x in, y out, the gradient of y in, that of x out; weights in and their gradients out
        return {"bytes": 4 * (4 * n * dim + 2 * mixer_weights), "flops": 6 * n * mixer_weights}
    weights = case["blocks"] * (mixer_weights + 3 * dim * FF[dim])
    n = B * (case["L"] if kind == "prefill" else 1)
    states = case["blocks"] * B * dim * 4 * (1 if kind == "prefill" else 2)
    # weights once at the precision of the matrix products, states, logits of one position per sequence
    return {"bytes": 2 * weights + states + 8 * n + 4 * B * VOCAB,
            "flops": 2 * n * weights + 2 * B * dim * VOCAB}


def tolerance(case):
    kind = case["kind"]
    if kind in ("prefill", "decode"):
        # up to 18 blocks of bfloat16 products on top of one another
        return {"rel": 2e-2}
    if kind == "mixer" or case.get("form") == "bf16" or case.get("dtype") == "bf16":
        return {"rel": 1e-2}
    return {"rel": 1e-5}
