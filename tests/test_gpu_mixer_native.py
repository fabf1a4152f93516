"""The native fused mixer (csrc/torch_mixer.cpp, field_rows.cuh, field_mixer_grad.cuh) against the same
mixer as a composition of torch operations, and the forward kernels at the edges of their tiles (GPU)."""
import numpy as np
import pytest
import torch

import mirror
from conftest import BF16_TOL, FP32_TOL, rel_err
from fields_lm_b200 import fused_field_read, fused_field_read_bf16, mixer
from oracle import field_oracle

pytestmark = pytest.mark.gpu


def _grads(m, x, gy, native):
    """y and every gradient, natively or through the composed path."""
    keep = mixer._native_mixer
    if not native:
        mixer._native_mixer = lambda *a: None
    try:
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = mixer.fused_mixer_forward(m, x)
    finally:
        mixer._native_mixer = keep
    assert ("FusedMixer" in type(y.grad_fn).__name__ or "FusedMixer" in y.grad_fn.name()) == native
    params = dict(m.named_parameters())
    grads = torch.autograd.grad(y, [x, *params.values()], gy)
    return {"y": y.detach(), "x": grads[0], **dict(zip(params, grads[1:]))}


# rows below, at and above one block of the gradient kernels, and of one warp or four per row; widths
# below, at and above one group of columns per thread
@pytest.mark.parametrize("dim,B,L", [(8, 1, 1), (64, 3, 7), (200, 2, 33), (1024, 2, 384), (1024, 5, 1003),
                                     (2048, 1, 65), (4096, 1, 70)])
def test_native_mixer_matches_the_composed_one(dim, B, L):
    torch.manual_seed(dim + L)
    m = mirror.IndependentVacancyField(dim).cuda()
    with torch.no_grad():
        m.read_norm.weight.add_(0.2 * torch.randn(2 * dim, device="cuda"))
        m.radius_logit.add_(torch.randn(dim // 2, device="cuda"))
        if dim >= 64:  # outside the clamp of the radius, where its gradient is zero
            m.radius_logit[0], m.radius_logit[1] = -1.0, 12.0
    x = torch.randn(B, L, dim, device="cuda", requires_grad=True)
    gy = torch.randn(B, L, dim, device="cuda")
    got, want = _grads(m, x, gy, True), _grads(m, x, gy, False)
    for name in want:
        assert got[name].shape == want[name].shape and got[name].dtype == want[name].dtype, name
        assert rel_err(got[name].float().cpu().numpy(), want[name].float().cpu().numpy()) < BF16_TOL, name


@pytest.mark.parametrize("dim", [200, 256])  # library products, fused ones
@pytest.mark.parametrize("which", ["x", "gradient", "both"])
def test_views_that_begin_anywhere(dim, which):
    """x and the incoming gradient as dense views one float into their storage: the results of aligned ones."""
    torch.manual_seed(dim)
    m = mirror.IndependentVacancyField(dim).cuda()

    def shifted(t):
        return torch.zeros(t.numel() + 1, device="cuda")[1:].view_as(t).copy_(t)

    x, gy = torch.randn(3, 37, dim, device="cuda"), torch.randn(3, 37, dim, device="cuda")
    want = _grads(m, x.clone().requires_grad_(), gy, True)
    x, gy = x if which == "gradient" else shifted(x), gy if which == "x" else shifted(gy)
    assert x.is_contiguous() and gy.is_contiguous() and bool(x.data_ptr() % 16 or gy.data_ptr() % 16)
    got = _grads(m, x.requires_grad_(), gy, True)
    for name in want:  # (the recurrence is reproducible to rounding)
        assert rel_err(got[name].float().cpu().numpy(), want[name].float().cpu().numpy()) < 2 ** -8, name


# widths and rows where fused and library products take turns, and where the columns of a thread of open_grad change
@pytest.mark.parametrize("dim,B,L", [(2048, 1, 3), (2056, 1, 40), (2064, 1, 4095), (2064, 1, 4096), (1024, 1, 129), (1032, 2, 301), (3072, 1, 4096),
                                     (3088, 1, 4096)])
def test_edges_of_the_rule(dim, B, L):
    test_native_mixer_matches_the_composed_one(dim, B, L)


# products with fused epilogues: several tiles of a pair, ragged rows, the widest; library products: a width that TMA does not
# address throughout, one beyond the rule
@pytest.mark.parametrize("dim,B,L", [(1024, 7, 1003), (1040, 1, 6145), (3072, 3, 2048), (1032, 3, 411), (2064, 1, 300)])
@pytest.mark.parametrize("x_grad", [True, False])
def test_mixer_with_fused_products(dim, B, L, x_grad):
    """... where x needs a gradient, and where it does not, which leaves the product of its gradient out."""
    torch.manual_seed(dim)
    m = mirror.IndependentVacancyField(dim).cuda()
    with torch.no_grad():
        m.read_norm.weight.add_(0.2 * torch.randn(2 * dim, device="cuda"))
    x = torch.randn(B, L, dim, device="cuda", requires_grad=x_grad)
    gy = torch.randn(B, L, dim, device="cuda")
    params, keep = dict(m.named_parameters()), mixer._native_mixer

    def run(native):
        mixer._native_mixer = keep if native else lambda *a: None
        try:
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = mixer.fused_mixer_forward(m, x)
        finally:
            mixer._native_mixer = keep
        assert ("FusedMixer" in y.grad_fn.name()) == native
        return [y.detach(), *torch.autograd.grad(y, ([x] if x_grad else []) + list(params.values()), gy)]

    for name, got, want in zip(["y"] + (["x"] if x_grad else []) + list(params), run(True), run(False)):
        assert got.shape == want.shape and got.dtype == want.dtype, name
        assert float((got - want).norm() / want.norm()) < BF16_TOL, name
        rows = want.flatten(0, -2) if want.dim() > 1 else want[None]  # (no row of a tile is off by itself)
        assert float(((got.view_as(rows) if rows.dim() > 1 else got) - rows).norm(dim=-1).max()) < BF16_TOL * float(rows.norm(dim=-1).max()), name


@pytest.mark.parametrize("L", [8, 9, 10, 35, 36, 37, 39, 40, 41, 79, 80, 81])
def test_forward_at_the_edges_of_the_tiles(L):
    rng = np.random.default_rng(L)
    B, C = 2, 132
    radius, theta = rng.uniform(0.5, 0.99995, C), rng.uniform(-np.pi, np.pi, C)
    par = [(radius * np.cos(theta)).astype(np.float32), (radius * np.sin(theta)).astype(np.float32),
           np.sqrt(np.maximum(1 - radius ** 2, 1e-4)).astype(np.float32)]
    raw = torch.from_numpy(rng.standard_normal((B, L, 3 * C)).astype(np.float32)).bfloat16()
    want, _ = field_oracle.forward(raw.float().numpy(), *par)
    dev = [torch.from_numpy(p).cuda() for p in par]
    assert rel_err(fused_field_read(raw.float().cuda(), *dev).cpu().numpy(), want) < FP32_TOL
    # one rounding to bfloat16 of values computed in fp32
    assert rel_err(fused_field_read_bf16(raw.cuda(), *dev).float().cpu().numpy(), want) < 2 ** -8


def test_bf16_forward_with_long_tiles():
    """Some thousand tiles of 40 steps in three channel groups."""
    B, L, C = 2, 35_003, 260
    torch.manual_seed(0)
    raw = (0.577 * torch.randn(B, L, 3 * C, device="cuda")).bfloat16()
    ring, theta = torch.linspace(0.85, 0.999, C), torch.linspace(0.03, 3.04, C)
    par = [t.cuda() for t in (ring * theta.cos(), ring * theta.sin(), (1 - ring ** 2).sqrt())]
    want = fused_field_read(raw.float(), *par)
    got = fused_field_read_bf16(raw, *par).float()
    assert float((got - want).abs().max()) <= 2 ** -8 * float(want.abs().max())


@pytest.mark.parametrize("plane", [0, 1, 2])
def test_nan_reaches_the_outputs(plane):
    """A NaN in one gate input or one token: from that step on in the operator's channel and in the mixer."""
    torch.manual_seed(plane)
    B, L, C, at, chan = 2, 150, 64, 70, 5
    ring, theta = torch.linspace(0.85, 0.999, C), torch.linspace(0.03, 3.04, C)
    par = [t.cuda() for t in (ring * theta.cos(), ring * theta.sin(), (1 - ring ** 2).sqrt())]
    raw = torch.randn(B, L, 3 * C, device="cuda")
    raw[1, at, plane * C + chan] = float("nan")
    want = fused_field_read(raw, *par).isnan().view(B, L, 4, C)
    got = fused_field_read_bf16(raw.bfloat16(), *par).isnan().view(B, L, 4, C)
    assert bool(want.any()) and bool((got == want).all())
    assert not bool(got[0].any() or got[1, :at].any() or got[..., torch.arange(C) != chan].any())
    m = mirror.IndependentVacancyField(2 * C).cuda()
    x = torch.randn(B, L, 2 * C, device="cuda")
    x[1, at, chan] = float("nan")
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        y = mixer.fused_mixer_forward(m, x)
    assert bool(y[1, at:].isnan().all()) and not bool(y[0].isnan().any() or y[1, :at].isnan().any())


def test_closed_gates_of_the_bf16_forward():
    """Vacancies down to the smallest and masks (lowest value, -inf): `read` is the fp32 one to its own rounding."""
    torch.manual_seed(3)
    C, closed = 64, [-40.0, -44.0, -45.0, -50.0, -60.0, -80.0, -100.0, -1e30, torch.finfo(torch.bfloat16).min, -torch.inf]
    ring, theta = torch.linspace(0.85, 0.999, C), torch.linspace(0.03, 3.04, C)
    par = [t.cuda() for t in (ring * theta.cos(), ring * theta.sin(), (1 - ring ** 2).sqrt())]
    raw = torch.randn(2, 60, 3 * C, device="cuda").bfloat16()
    raw[:, 3:, 2 * C:] = torch.tensor(closed, device="cuda").repeat(400)[:57 * C].view(57, C).bfloat16()
    want = fused_field_read(raw.float(), *par)
    got = fused_field_read_bf16(raw, *par).float()
    assert bool((want[:, 3:, 2 * C:] == 0).any()) and bool((got[want == 0] == 0).all())
    assert bool(((got - want).abs() <= (2 ** -8 * want.abs()).clamp_min(2.0 ** -126)).all())


def test_state_of_the_bf16_forward_is_as_accurate_as_the_fp32_one():
    """The state stays fp32 on the bfloat16 boundary: its error against 64 bits is the fp32 operator's."""
    from fields_lm_b200 import _lib, field_read_with_state
    lib, (B, L, C) = _lib.load(), (8, 500, 512)
    torch.manual_seed(4)
    ring, theta = torch.linspace(0.85, 0.999, C), torch.linspace(0.03, 3.04, C)
    par = [t.cuda() for t in (ring * theta.cos(), ring * theta.sin(), (1 - ring ** 2).sqrt())]
    raw = (0.577 * torch.randn(B, L, 3 * C, device="cuda")).bfloat16()
    _, want = field_oracle.forward(raw.float().cpu().numpy(), *[p.cpu().numpy() for p in par])
    want = torch.from_numpy(np.asarray(want, dtype=np.float64)).cuda()
    read, state = torch.empty(B, L, 4 * C, device="cuda", dtype=torch.bfloat16), torch.empty(B, 2 * C, device="cuda")
    n = lib.fields_read_workspace_bytes(B, L, C, 0)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    assert lib.fields_read_forward_bf16(raw.data_ptr(), *[p.data_ptr() for p in par], None, read.data_ptr(), state.data_ptr(),
                                        ws.data_ptr(), n, B, L, C, torch.cuda.current_stream().cuda_stream) == 0
    err = [float((s.double() - want).norm() / want.norm()) for s in (state, field_read_with_state(raw.float(), *par)[1])]
    assert err[0] < 1.15 * err[1], err  # (1.3e-7 both; 1.9e-7 with one reciprocal shared by the three gates)


def test_open_gates_of_the_bf16_forward():
    """The recurrence inside a tile takes the keep factor of the maps between tiles: a state that only decays (lambda = 1),
    in the sums of squares of ten steps against the end states of one and of ten."""
    from fields_lm_b200 import _lib
    lib, B, L, C = _lib.load(), 320, 10, 4
    raw = torch.zeros(B, L, 3 * C, device="cuda", dtype=torch.bfloat16)
    raw[:, 0, :C] = 1.0
    raw[..., 2 * C:] = (3 + torch.arange(B, device="cuda") / 64)[:, None, None]  # open gates, one per row of the batch
    one, zero = torch.ones(C, device="cuda"), torch.zeros(C, device="cuda")

    def call(steps):
        read = torch.empty(B, steps, 4 * C, device="cuda", dtype=torch.bfloat16)
        state, sums = torch.empty(B, 2 * C, device="cuda"), torch.empty(B, steps, 1, device="cuda")
        n, x = lib.fields_read_workspace_bytes(B, steps, C, 0), raw[:, :steps].contiguous()
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        assert lib.fields_read_forward_bf16_stats(*[t.data_ptr() for t in (x, one, zero, one)], None, read.data_ptr(), sums.data_ptr(),
                                                  state.data_ptr(), ws.data_ptr(), n, B, steps, C,
                                                  torch.cuda.current_stream().cuda_stream) == 0
        return state[:, 0].double(), sums[..., 0].double()

    (first, _), (last, sums) = call(1), call(L)
    keep = (last / first) ** (1 / (L - 1))
    k = torch.arange(L - 1, device="cuda")
    off = (sums[:, 1:] / (sums[:, 1:2] * keep[:, None] ** (2 * k)) - 1).abs()
    # squared twice the relative error: of the product of each step in the recurrence and in the map behind `keep`, three in the
    # squares and their sum
    assert bool((off <= 2.0 ** -24 * (4 * k + 6)).all()), off.amax(0)


@pytest.mark.parametrize("wanted", [("x",), ("x", "write_proj.bias"), ("gate_proj.weight",), ("write_proj.weight",),
                                    ("out_proj.weight", "gate_proj.bias"), ("read_norm.weight",), ("radius_logit",),
                                    ("theta", "out_proj.bias"), ("write_proj.weight", "gate_proj.weight")])
@pytest.mark.parametrize("D", [1024, 1032])  # products with fused epilogues, the library's
def test_frozen_parameters_cost_nothing(wanted, D):
    """Gradients of some inputs alone are those of the full pass, and what only the others need is not computed: a
    third of the weights' gradients is more than the difference that the allocator sees."""
    torch.manual_seed(6)
    B, L = 1, 40
    m = mirror.IndependentVacancyField(D).cuda()
    x = torch.randn(B, L, D, device="cuda", requires_grad=True)
    gy = torch.randn(B, L, D, device="cuda")
    full = _grads(m, x, gy, True)
    leaves = {"x": x, **dict(m.named_parameters())}

    def backward():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = mixer.fused_mixer_forward(m, x)
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        needed = [t for t in leaves.values() if t.requires_grad]
        got = torch.autograd.grad(y, needed, gy)
        torch.cuda.synchronize()
        return dict(zip([n for n, t in leaves.items() if t.requires_grad], got)), torch.cuda.max_memory_allocated() - before

    _, most = backward()
    for name, t in leaves.items():
        t.requires_grad_(name in wanted)
    got, peak = backward()
    for name in wanted:
        assert torch.equal(got[name], full[name]) or rel_err(got[name].cpu().numpy(), full[name].cpu().numpy()) < 1e-6
    sizes = {"write_proj.weight": 3 * D * D // 2, "gate_proj.weight": D * D, "out_proj.weight": 2 * D * D}
    spared = sum(n for name, n in sizes.items()
                 if name not in wanted and not (name == "out_proj.weight" and "read_norm.weight" in wanted))
    assert peak <= most - 4 * spared * 0.9


@pytest.mark.parametrize("name", ["radius_logit", "theta"])
def test_nan_parameters_reach_the_outputs(name):
    """A NaN in the transition of one channel: the output and the gradients of that channel are NaN, as composed."""
    torch.manual_seed(7)
    m = mirror.IndependentVacancyField(64).cuda()
    with torch.no_grad():
        getattr(m, name)[5] = float("nan")
    x = torch.randn(1, 20, 64, device="cuda", requires_grad=True)
    gy = torch.randn_like(x)
    got, want = _grads(m, x, gy, True), _grads(m, x, gy, False)
    assert bool(want["y"].isnan().all()) and bool(want[name][5].isnan())
    for key in want:
        assert torch.equal(got[key].isnan(), want[key].isnan()), key
