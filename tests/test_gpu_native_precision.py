"""The native mixer, prefill and step are no further from 64-bit arithmetic than the same model module by module under
bfloat16 autocast (GPU)."""
import copy

import pytest
import torch
import torch.nn.functional as F

import mirror
from test_gpu_mixer_native import _grads
from test_gpu_stack import LM, _run

pytestmark = pytest.mark.gpu

# Both paths round the same operands to bfloat16 as often, so their errors are nearly equal: measured 0.73 to 1.013 of
# the modules' over these sizes.
FACTOR = 1.1


def _read(raw, tr, ti, gamma, state):
    C, out = tr.numel(), []
    zr, zi, zv = raw.split(C, -1)
    jr, ji, v = torch.tanh(zr), torch.tanh(zi), 0.9 * torch.sigmoid(zv)
    sr, si = state.split(C, -1)
    for t in range(raw.shape[1]):
        mr, mi, vt = tr * sr - ti * si, tr * si + ti * sr, v[:, t]
        sr, si = (1 - vt) * mr + gamma * vt * jr[:, t], (1 - vt) * mi + gamma * vt * ji[:, t]
        out.append(torch.cat([sr, si, vt * mr, vt * mi], -1))
    return torch.stack(out, 1), torch.cat([sr, si], -1)


def _norm(n, x):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + n.eps) * n.weight


def _mixer(m, x, state):
    radius = torch.sigmoid(m.radius_logit).clamp(0.50, 0.99995)
    par = radius * torch.cos(m.theta), radius * torch.sin(m.theta), torch.sqrt((1 - radius.square()).clamp_min(1e-4))
    read, state = _read(m.write_proj(x), *par, state)
    return x + m.out_proj(_norm(m.read_norm, read)) * torch.sigmoid(m.gate_proj(x)), state


def _block(b, x, state):
    x, state = _mixer(b.mixer, x, state)
    u, v = b.ff.w12(_norm(b.ff_norm, x)).chunk(2, -1)
    return x + b.ff.w3(F.silu(u) * v), state


def _err(a, want):
    return float((a.double() - want).norm() / want.norm())


@pytest.mark.parametrize("dim,B,L", [(1024, 2, 300), (256, 1, 64), (512, 8, 33)])
def test_mixer(dim, B, L):
    torch.manual_seed(dim)
    m = mirror.IndependentVacancyField(dim).cuda()
    with torch.no_grad():
        for p in m.parameters():
            p.add_(0.05 * torch.randn_like(p) if p.dim() == 1 else 0)
    x = torch.randn(B, L, dim, device="cuda", requires_grad=True)
    gy = torch.randn(B, L, dim, device="cuda")
    native, modules = _grads(m, x, gy, True), _grads(m, x, gy, False)
    m64, x64 = copy.deepcopy(m).double(), x.detach().double().requires_grad_(True)
    y, _ = _mixer(m64, x64, x64.new_zeros(B, dim))
    params = dict(m64.named_parameters())
    want = {"y": y.detach(), **dict(zip(["x", *params], torch.autograd.grad(y, [x64, *params.values()], gy.double())))}
    for name, w in want.items():
        assert _err(native[name], w) < FACTOR * _err(modules[name], w), name


@pytest.mark.parametrize("dim,hidden,layers,B,L", [(1024, 2528, 8, 8, 64), (512, 1344, 8, 1, 200), (256, 704, 4, 16, 16),
                                                   (512, 1344, 4, 600, 3)])
def test_prefill_and_step(dim, hidden, layers, B, L):
    torch.manual_seed(dim + B)
    model = LM(dim, layers, hidden).cuda()
    for p in model.parameters():  # norm weights away from one
        if p.dim() == 1 and p.numel() in (dim, 2 * dim):
            p.data += 0.1 * torch.randn_like(p)
    tokens = torch.randint(0, 97, (B, L + 3), device="cuda")
    native, modules = _run(model, tokens, L, True), _run(model, tokens, L, False)
    m64 = copy.deepcopy(model).double()
    logits = []
    with torch.no_grad():
        states = [torch.zeros(B, dim, device="cuda", dtype=torch.float64) for _ in m64.blocks]
        for piece in [tokens[:, :L], *tokens[:, L:].split(1, 1)]:
            x = m64.emb(piece)
            for i, b in enumerate(m64.blocks):
                x, states[i] = _block(b, x, states[i])
            logits.append(m64.lm_head(_norm(m64.final_norm, x[:, -1])))
    for a, b, want in zip(native[0], modules[0], logits):
        assert _err(a, want) < FACTOR * _err(b, want)
    a, b, want = (torch.cat(list(s)) for s in (native[1].states, modules[1].states, states))
    assert _err(a, want) < FACTOR * _err(b, want)


def test_mixer_with_fused_products():
    test_mixer(640, 8, 800)


def test_prefill_with_fused_products():
    test_prefill_and_step(1024, 2528, 4, 8, 256)
