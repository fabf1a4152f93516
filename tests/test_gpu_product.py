"""fields_product, the products with fused epilogues (csrc/field_product.cuh), and the layouts of their weights, through the
C ABI against the same formulas in 64 bits (GPU)."""
import ctypes

import pytest
import torch

from fields_lm_b200 import _lib

pytestmark = pytest.mark.gpu
P, LL, I, F = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_float
BIAS, GATE, SWIGLU, RESIDUAL, NORM_GRAD = range(5)


class Args(ctypes.Structure):
    _fields_ = [("a", P), ("b", P), ("rows", LL), ("cols", I), ("depth", I), ("x", P), ("bias", P), ("gate_bias", P), ("sums", P),
                ("row", P), ("bias16", P), ("gate", P), ("read", P), ("gate_pitch", LL), ("h_pitch", LL), ("entries", I),
                ("features", I), ("eps", F), ("y", P), ("sums_out", P), ("h", P), ("acc", P)]


def _stream():
    return torch.cuda.current_stream().cuda_stream


# one row; rows, columns and depth around the edges of a warp's piece, of a block's tile and of a k-block; one tile and
# several rounds of tiles, of 128 and of 256 columns
@pytest.mark.parametrize("kind", range(5))
@pytest.mark.parametrize("M,N,K", [(1, 16, 16), (31, 48, 72), (129, 144, 64), (257, 272, 1000), (300, 1024, 2528), (4100, 5056, 1024),
                                   (12000, 1040, 200), (20000, 256, 136)])
def test_product(kind, M, N, K):
    torch.manual_seed(M + N + kind)
    dev, pitch = "cuda", N + 8

    def rand(*shape):
        return torch.randn(*shape, device=dev)

    def halves(width):  # rows of a wider matrix
        return torch.full((M, pitch), float("nan"), device=dev, dtype=torch.bfloat16)[:, :width]

    t = dict(a=rand(M, K).bfloat16(), b=(rand(N, K) / K ** 0.5).bfloat16())
    d = {}
    out = t["a"].double() @ t["b"].double().T
    entries, features, eps = {31: 4, 257: 32, 4100: 36}.get(M, 3), 100, 1e-3
    sums = rand(M, entries).square() * 30
    rstd = torch.rsqrt(sums.double().sum(1, keepdim=True) / features + eps)
    if kind == BIAS:
        t.update(bias16=rand(N).bfloat16(), h=halves(N))
        d["h"] = out + t["bias16"].double()
    if kind == GATE:
        x = rand(M, N)
        gate = halves(N).copy_(rand(M, N))
        t.update(x=x.clone(), bias=rand(N), gate_bias=rand(N), gate=gate, sums=sums, h=halves(N),
                 acc=torch.empty(M, N, device=dev, dtype=torch.bfloat16), sums_out=torch.empty(M, (N + 31) // 32, device=dev))
        t["y"] = t["x"]  # in place
        y = x.double() + (out * rstd + t["bias"].double()) * torch.sigmoid(gate.double() + t["gate_bias"].double())
        d.update(y=y, h=y, acc=out)
    if kind == SWIGLU:
        t.update(sums=sums, h=halves(N // 2))
        uv = (out * rstd).view(M, N // 16, 2, 8)
        d["h"] = torch.nn.functional.silu(uv[:, :, 0]).mul(uv[:, :, 1]).reshape(M, N // 2)
    if kind == RESIDUAL:
        t.update(x=rand(M, N), y=torch.empty(M, N, device=dev), h=halves(N))
        d["y"] = d["h"] = t["x"].double() + out
    if kind == NORM_GRAD:
        t.update(read=rand(M, N).bfloat16(), row=rand(M), h=halves(N))
        d["h"] = out + 2 * t["row"].double()[:, None] * t["read"].double()
    args = Args(rows=M, cols=N, depth=K, gate_pitch=pitch, h_pitch=pitch, entries=entries, features=features, eps=eps,
                **{k: v.data_ptr() for k, v in t.items()})
    assert _lib.load().fields_product(ctypes.byref(args), kind, _stream()) == 0
    torch.cuda.synchronize()
    for name, want in d.items():
        # one rounding to bfloat16 is 2^-9 of each value; fp32 sums of K products err by less than 1e-5 in the norm
        err = float((t[name].double() - want).norm() / want.norm())
        assert err < (2 ** -8 if t[name].dtype == torch.bfloat16 else 1e-5), (name, err)
        # and value by value: sums of K products of about 1 / sqrt(K) err by less than 1e-4 of a value's usual size
        bound = 1e-4 * want.square().mean().sqrt() + (2 ** -8 * want.abs() if t[name].dtype == torch.bfloat16 else 0)
        assert bool(((t[name].double() - want).abs() <= bound).all()), name
    if kind == GATE:
        want = d["y"].square().sum(1)
        assert float(((t["sums_out"].double().sum(1) - want).abs() / want).max()) < 1e-4
    if "h" in t:  # nothing beside the columns
        whole = torch.as_strided(t["h"], (M, pitch), (pitch, 1))
        assert bool(whole[:, t["h"].shape[1]:].isnan().all())


def test_refusals():
    lib, a = _lib.load(), torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    ok = dict(a=a.data_ptr(), b=a.data_ptr(), rows=8, cols=16, depth=16, bias16=a.data_ptr(), h=a.data_ptr(), h_pitch=64)
    assert lib.fields_product(None, BIAS, _stream()) == 1
    for bad, rc in ((dict(b=None), 1), (dict(cols=0), 1), (dict(h=None), 1), (dict(depth=12), 2), (dict(a=a.data_ptr() + 2), 2),
                    (dict(h_pitch=63), 2)):
        assert (lib.fields_product(ctypes.byref(Args(**{**ok, **bad})), BIAS, _stream()) != 0) == bool(rc), bad
    assert lib.fields_product(ctypes.byref(Args(**ok)), 5, _stream()) != 0
    assert lib.fields_product(ctypes.byref(Args(**{**ok, "rows": 0})), BIAS, _stream()) == 0


@pytest.mark.parametrize("kind", [BIAS, GATE, SWIGLU])
def test_pitches(kind):
    """None is dense; one that makes rows overlap or that 32 bits do not address is refused."""
    M, N, K, lib = 5, 32, 16, _lib.load()
    torch.manual_seed(kind)
    width = N // 2 if kind == SWIGLU else N

    def rand(*shape):
        return torch.randn(*shape, device="cuda")

    t = dict(a=rand(M, K).bfloat16(), b=rand(N, K).bfloat16(), bias16=rand(N).bfloat16(), x=rand(M, N), bias=rand(N),
             gate_bias=rand(N), gate=rand(M, N).bfloat16(), sums=rand(M, 3).square())

    def call(**pitches):
        h, y = torch.full((M, width), float("nan"), device="cuda", dtype=torch.bfloat16), torch.empty(M, N, device="cuda")
        args = Args(rows=M, cols=N, depth=K, entries=3, features=10, eps=1e-3, h=h.data_ptr(), y=y.data_ptr(),
                    **{k: v.data_ptr() for k, v in t.items()}, **pitches)
        rc = lib.fields_product(ctypes.byref(args), kind, _stream())
        torch.cuda.synchronize()
        return rc, h

    (rc, got), (rc2, want) = call(), call(gate_pitch=N, h_pitch=width)
    assert rc == rc2 == 0 and torch.equal(got, want) and not bool(want.isnan().any())
    refused = [dict(h_pitch=width - 4), dict(h_pitch=4), dict(h_pitch=-width), dict(h_pitch=(1 << 26) + 4)]
    if kind == GATE:
        refused += [dict(gate_pitch=N - 4), dict(gate_pitch=-N), dict(gate_pitch=(1 << 26) + 4)]
    for pitches in refused:
        rc, h = call(**pitches)
        assert rc != 0 and bool(h.isnan().all()), pitches


# one row, the edges of a warp's 32 rows and of its 32 or 64 columns, several tiles of a pair
@pytest.mark.parametrize("kind", range(5))
@pytest.mark.parametrize("M,N,K", [(1, 16, 16), (33, 80, 72), (97, 272, 200), (12000, 1040, 72)])
def test_rows_that_tma_does_not_address(kind, M, N, K):
    """bfloat16 rows that lie on 8 bytes only give the same bits as aligned ones; so do N - 4 columns, and acc without h."""
    torch.manual_seed(M + kind)
    lib = _lib.load()

    def rand(*shape):
        return torch.randn(*shape, device="cuda")

    whole = dict(a=rand(M, K).bfloat16(), b=rand(N, K).bfloat16(), bias16=rand(N).bfloat16(), x=rand(M, N), bias=rand(N),
                 gate_bias=rand(N), gate=rand(M, N).bfloat16(), sums=rand(M, 3).square(), read=rand(M, N).bfloat16(), row=rand(M))

    def call(n, shift, h=True):
        width = n // 2 if kind == SWIGLU else n
        t = {k: v[:, :n].contiguous() if k in ("x", "read") else v for k, v in whole.items()}
        pitch = n + 8 + shift

        def halves(cols):  # rows `shift` elements off 16 bytes
            return torch.full((M * pitch + 8,), float("nan"), device="cuda", dtype=torch.bfloat16)[shift:shift + M * pitch].view(
                M, pitch)[:, :cols]

        t["gate"] = halves(n).copy_(whole["gate"][:, :n])
        out = dict(y=rand(M, n), acc=torch.full((M, n), float("nan"), device="cuda", dtype=torch.bfloat16),
                   sums_out=torch.zeros(M, (n + 31) // 32, device="cuda"), h=halves(width) if h else None)
        args = Args(rows=M, cols=n, depth=K, entries=3, features=10, eps=1e-3, gate_pitch=pitch, h_pitch=pitch,
                    **{k: v.data_ptr() for k, v in {**t, **out}.items() if v is not None})
        assert lib.fields_product(ctypes.byref(args), kind, _stream()) == 0
        torch.cuda.synchronize()
        names = {GATE: ("y", "acc", "h"), RESIDUAL: ("y", "h")}.get(kind, ("h",))
        return {k: out[k] for k in names if out[k] is not None}, out["sums_out"]

    want, sums = call(N, 0)
    assert not any(bool(v.isnan().any()) for v in want.values())
    got, got_sums = call(N, 4)
    assert all(torch.equal(got[k], want[k]) for k in want) and torch.equal(got_sums, sums)
    if kind != SWIGLU:  # (of u and v in turn no four columns can go)
        got, _ = call(N - 4, 0)
        assert all(torch.equal(got[k], want[k][:, :N - 4]) for k in want)
    if kind in (GATE, RESIDUAL):
        got, _ = call(N, 0, h=False)
        assert all(torch.equal(got[k], want[k]) for k in got)


# the same sizes; the input alone or the output alone lies on 8 bytes
@pytest.mark.parametrize("kind", [BIAS, GATE, NORM_GRAD])
@pytest.mark.parametrize("M,N,K", [(1, 16, 16), (33, 80, 72), (97, 272, 200), (12000, 1040, 72)])
def test_one_of_the_tensors_that_tma_does_not_address(kind, M, N, K):
    """... gives the same bits as both aligned, and what lies between the rows stays as it was."""
    torch.manual_seed(M + kind)
    lib = _lib.load()

    def rand(*shape):
        return torch.randn(*shape, device="cuda")

    t = dict(a=rand(M, K).bfloat16(), b=rand(N, K).bfloat16(), bias16=rand(N).bfloat16(), x=rand(M, N), bias=rand(N),
             gate_bias=rand(N), sums=rand(M, 3).square(), row=rand(M))
    values = rand(M, N).bfloat16()

    def off(pitch, shift):
        return torch.full((M * pitch + 8,), float("nan"), device="cuda", dtype=torch.bfloat16)[shift:shift + M * pitch].view(M, pitch)

    def call(in_shift, out_shift):
        gate, read, h, y = off(N + 8 + in_shift, in_shift), off(N, in_shift), off(N + 8 + out_shift, out_shift), rand(M, N)
        gate[:, :N].copy_(values)
        read.copy_(values)
        args = Args(rows=M, cols=N, depth=K, entries=3, features=10, eps=1e-3, gate_pitch=gate.stride(0), h_pitch=h.stride(0),
                    y=y.data_ptr(), h=h.data_ptr(), gate=gate.data_ptr(), read=read.data_ptr(), **{k: v.data_ptr() for k, v in t.items()})
        assert lib.fields_product(ctypes.byref(args), kind, _stream()) == 0
        torch.cuda.synchronize()
        assert bool(h[:, N:].isnan().all())
        return [h[:, :N], y] if kind == GATE else [h[:, :N]]

    want = call(0, 0)
    assert not any(bool(v.isnan().any()) for v in want)
    for shifts in [(4, 0), (0, 4)]:
        assert all(torch.equal(a, b) for a, b in zip(call(*shifts), want)), shifts


# columns and depth around the edges of 64 (a box of the weights), of both tile widths; several tiles of a pair
@pytest.mark.parametrize("kind", [RESIDUAL, NORM_GRAD])
@pytest.mark.parametrize("M,N,K", [(1, 16, 16), (130, 72, 64), (257, 200, 136), (300, 1024, 2528), (16000, 272, 72), (9000, 1024, 200)])
def test_weights_by_depth(kind, M, N, K):
    torch.manual_seed(M + kind)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(K, N, device="cuda") / K ** 0.5).bfloat16()
    x, row = torch.randn(M, N, device="cuda"), torch.randn(M, device="cuda")
    read, h = torch.randn(M, N, device="cuda").bfloat16(), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    y = torch.empty(M, N, device="cuda")
    args = Args(rows=M, cols=N, depth=K, **{k: v.data_ptr() for k, v in dict(a=a, b=b, x=x, row=row, read=read, h=h, y=y).items()})
    assert _lib.load().fields_product(ctypes.byref(args), kind + 16, _stream()) == 0
    torch.cuda.synchronize()
    want = a.double() @ b.double() + (x.double() if kind == RESIDUAL else 2 * row.double()[:, None] * read.double())
    for got in (h, y) if kind == RESIDUAL else (h,):
        # (as above: a rounding to bfloat16, and fp32 sums of K products)
        bound = 1e-4 * want.square().mean().sqrt() + (2 ** -8 * want.abs() if got is h else 0)
        assert bool(((got.double() - want).abs() <= bound).all())


def test_weights_by_depth_refusals():
    lib, a = _lib.load(), torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    args = Args(rows=8, cols=12, depth=16, **{k: a.data_ptr() for k in ("a", "b", "x", "y", "bias16", "h", "read", "row")})
    assert lib.fields_product(ctypes.byref(args), RESIDUAL, _stream()) == 0
    assert lib.fields_product(ctypes.byref(args), RESIDUAL + 16, _stream()) != 0  # rows of 24 bytes
    args.cols = 16
    for kind in (BIAS, GATE, SWIGLU):
        assert lib.fields_product(ctypes.byref(args), kind + 16, _stream()) != 0


class Transpose(ctypes.Structure):
    _fields_ = [("in_", P), ("out", P), ("rows", I), ("cols", I)]


@pytest.mark.parametrize("shapes", [[(2, 2)], [(62, 64), (66, 130)], [(1024, 2048), (2560, 1024)], [(16, 40)]])
def test_transpose(shapes):
    ins = [torch.randn(s, device="cuda").bfloat16() for s in shapes]
    outs = [torch.zeros(s[::-1], device="cuda", dtype=torch.bfloat16) for s in shapes]
    parts = (Transpose * len(ins))(*[Transpose(i.data_ptr(), o.data_ptr(), *i.shape) for i, o in zip(ins, outs)])
    assert _lib.load().fields_transpose_bf16(parts, len(ins), _stream()) == 0
    torch.cuda.synchronize()
    assert all(torch.equal(o, i.T) for i, o in zip(ins, outs))


@pytest.mark.parametrize("D,H", [(16, 8), (64, 40), (1024, 2528)])
def test_w12_in_parts(D, H):
    """w12 by itself, as it is and in the order of the fused products, which is that of the step."""
    from test_gpu_step_block import StackWeights, StepWeights
    lib, C = _lib.load(), D // 2
    torch.manual_seed(D)
    rows = lib.fields_step_w12_rows(H)
    f32 = {n: torch.randn(s, device="cuda") for n, s in dict(
        write_w=(3 * C, D), write_b=(3 * C,), gate_w=(D, D), gate_b=(D,), out_w=(D, 2 * D), read_norm_w=(2 * D,),
        w12=(2 * H, D), w3=(D, H), radius_logit=(C,), theta=(C,), par=(3, C), norm=(D,), in_b32=(5 * C,)).items()}
    b16 = {n: torch.zeros(s, device="cuda", dtype=torch.bfloat16) for n, s in dict(
        in_w=(5 * C, D), in_b=(5 * C,), out_w16=(D, 2 * D), w3_16=(D, H), plain=(2 * H, D), order=(2 * H, D), step=(rows, D),
        step_in=(5 * C, D)).items()}
    a = {n: t.data_ptr() for n, t in {**f32, **b16}.items()}

    def weights(w12_16):
        return StackWeights(a["write_w"], a["write_b"], a["gate_w"], a["out_w"], a["read_norm_w"], a["w12"], a["w3"],
                            a["radius_logit"], a["theta"], a["in_w"], a["in_b"], a["out_w16"], w12_16, a["w3_16"], a["par"], D, H)

    norms = (P * 1)(a["norm"])
    assert lib.fields_stack_layout_parts(ctypes.byref(weights(None)), None, 1, 1, _stream()) == 0
    assert lib.fields_stack_layout_parts(ctypes.byref(weights(a["plain"])), None, 1, 2, _stream()) == 0
    assert lib.fields_stack_layout_parts(ctypes.byref(weights(a["order"])), norms, 1, 4, _stream()) == 0
    step = StepWeights(a["write_w"], a["write_b"], a["gate_w"], a["gate_b"], a["w12"], a["norm"], a["step_in"], a["step"], a["in_b32"],
                       D, H)
    assert lib.fields_step_layout(ctypes.byref(step), _stream()) == 0
    torch.cuda.synchronize()
    assert torch.equal(b16["plain"], f32["w12"].bfloat16()) and torch.equal(b16["w3_16"], f32["w3"].bfloat16())
    assert torch.equal(b16["order"], b16["step"][:2 * H])
    u, v = (f32["w12"] * f32["norm"]).bfloat16().view(2, H // 8, 8, D)
    assert torch.equal(b16["order"].view(H // 8, 2, 8, D), torch.stack([u, v], 1))
