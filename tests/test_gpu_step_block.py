"""fields_step_block and fields_step_stack through the C ABI (GPU)."""
import ctypes

import pytest
import torch

from fields_lm_b200 import _lib

pytestmark = pytest.mark.gpu
P, F, I = ctypes.c_void_p, ctypes.c_float, ctypes.c_int


def _struct(name, *fields):
    return type(name, (ctypes.Structure,), {"_fields_": list(fields)})


StackWeights = _struct("StackWeights", *[(n, P) for n in (
    "write_w", "write_b", "gate_w", "out_w", "read_norm_w", "w12", "w3", "radius_logit", "theta",
    "in_w", "in_b", "out_w16", "w12_16", "w3_16", "par")], ("dim", I), ("hidden", I))
StepWeights = _struct("StepWeights", *[(n, P) for n in (
    "write_w", "write_b", "gate_w", "gate_b", "w12", "ff_norm_w", "in_w", "w12_w", "in_b")], ("dim", I), ("hidden", I))
StepArgs = _struct("StepArgs", *[(n, P) for n in (
    "x", "state", "y", "xb", "yb", "read", "gate", "act", "read_sq", "y_sq", "in_w", "out_w16", "w12_w", "w3_16",
    "in_b", "par", "out_b")], ("read_eps", F), ("ff_eps", F), ("rows", I), ("dim", I), ("hidden", I), ("settled", I))


@pytest.mark.parametrize("M,D,H", [(16, 1024, 2528), (128, 512, 1344)])
def test_step_block_waits_for_the_layout_it_follows(M, D, H):
    lib, C = _lib.load(), D // 2
    torch.manual_seed(M)
    rows = lib.fields_step_w12_rows(H)
    f32 = dict(write_w=(3 * C, D), write_b=(3 * C,), gate_w=(D, D), gate_b=(D,), out_w=(D, 2 * D), out_b=(D,),
               read_norm_w=(2 * D,), ff_norm_w=(D,), w12=(2 * H, D), w3=(D, H), radius_logit=(C,), theta=(C,), par=(3, C),
               in_b32=(5 * C,), x=(M, D), y=(M, D), state=(M, D), read_sq=(C // 8, M), y_sq=(D // 8, M))
    b16 = dict(in_w=(5 * C, D), in_full=(5 * C, D), in_b=(5 * C,), out_w16=(D, 2 * D), w12_16=(2 * H, D), w3_16=(D, H),
               w12_w=(rows, D), xb=(M, D), yb=(M, D), read=(M, 2 * D), gate=(M, D), act=(M, H))
    t = {n: torch.randn(s, device="cuda") / s[-1] ** 0.5 for n, s in f32.items()}
    t.update({n: torch.zeros(s, device="cuda", dtype=torch.bfloat16) for n, s in b16.items()})
    a = {n: v.data_ptr() for n, v in t.items()}
    stack = StackWeights(*[a[n] for n in ("write_w", "write_b", "gate_w", "out_w", "read_norm_w", "w12", "w3", "radius_logit",
                                          "theta", "in_full", "in_b", "out_w16", "w12_16", "w3_16", "par")], D, H)
    step = StepWeights(*[a[n] for n in ("write_w", "write_b", "gate_w", "gate_b", "w12", "ff_norm_w", "in_w", "w12_w",
                                        "in_b32")], D, H)
    args = StepArgs(*[a[n] for n in ("x", "state", "y", "xb", "yb", "read", "gate", "act", "read_sq", "y_sq", "in_w",
                                     "out_w16", "w12_w", "w3_16", "in_b32", "par", "out_b")], 1e-6, 1e-6, M, D, H, 0)
    stream = torch.cuda.current_stream().cuda_stream
    state = t["state"].clone()

    def block(wait):
        t["xb"].copy_(t["x"])
        t["state"].copy_(state)
        assert lib.fields_stack_layout(ctypes.byref(stack), 1, stream) == 0
        assert lib.fields_step_layout(ctypes.byref(step), stream) == 0
        if wait:
            torch.cuda.synchronize()
        assert lib.fields_step_block(ctypes.byref(args), stream) == 0
        torch.cuda.synchronize()
        return t["y"].clone(), t["state"].clone()

    for i in range(10):  # other weights every time: what was laid out before is no help
        for n in ("write_w", "gate_w", "out_w", "w12", "w3", "write_b", "theta"):
            t[n].mul_(-1.0 if i % 2 else 1.1)
        got, want = block(False), block(True)
        assert all(torch.equal(g, w) for g, w in zip(got, want))
        assert not bool(got[0].isnan().any())


# rows at the edges of a row tile and of the share of a row tile that a block of a cluster finishes, up to four row
# tiles; widths with few and many column tiles; more blocks than one launch takes
@pytest.mark.parametrize("M,D,H,blocks", [(1, 64, 8, 26), (3, 272, 360, 2), (127, 16, 24, 3), (129, 1024, 2528, 2),
                                          (200, 512, 1344, 3), (257, 256, 704, 2), (512, 1024, 704, 2), (5, 2048, 96, 2)])
def test_step_stack_is_its_phases_one_by_one(M, D, H, blocks):
    """One launch whose blocks wait for one another computes bit for bit what a launch per product does."""
    lib, C = _lib.load(), D // 2
    torch.manual_seed(M + D)

    def bf16(*shape):
        return (torch.randn(shape, device="cuda") / shape[-1] ** 0.5).bfloat16()

    weights = [dict(in_w=bf16(5 * C, D), out_w16=bf16(D, 2 * D), w12_w=bf16(lib.fields_step_w12_rows(H), D), w3_16=bf16(D, H),
                    in_b=torch.randn(5 * C, device="cuda"), par=torch.rand(3, C, device="cuda"),
                    out_b=torch.randn(D, device="cuda")) for _ in range(blocks)]
    x0, state0 = torch.randn(M, D, device="cuda"), torch.randn(blocks, M, D, device="cuda")

    def run(one_launch):
        x, state = x0.clone(), state0.clone()
        scratch = dict(y=torch.empty_like(x), xb=x.bfloat16(), yb=bf16(M, D), read=bf16(M, 2 * D), gate=bf16(M, D), act=bf16(M, H),
                       read_sq=torch.empty(C // 8, M, device="cuda"), y_sq=torch.empty(D // 8, M, device="cuda"))
        args = (StepArgs * blocks)()
        for i, w in enumerate(weights):
            given = {n: t.data_ptr() for n, t in {**scratch, **w}.items()}
            given.update(x=(x if i == 0 else scratch["y"]).data_ptr(), state=state[i].data_ptr())
            args[i] = StepArgs(*[given[n] for n, _ in StepArgs._fields_[:17]], 1e-6, 1e-5, M, D, H, 0)
        sync = torch.empty(512, dtype=torch.uint8, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        assert lib.fields_step_stack(args, blocks, sync.data_ptr() if one_launch else None, stream) == 0
        torch.cuda.synchronize()
        return scratch["y"], scratch["xb"], state

    got, want = run(True), run(False)
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and not bool(want[0].isnan().any())


# one row; rows and widths at the edges of a tile; K in one part, in as many as a cluster has blocks, and in fewer than fit
# the GPU (384 rows); feed-forward widths that leave part of a tile; wide and narrow tiles
@pytest.mark.parametrize("M,D,H", [(1, 16, 8), (3, 272, 360), (128, 48, 24), (127, 64, 176), (384, 384, 960), (129, 1024, 2528),
                                   (512, 256, 704), (5, 2048, 96), (300, 768, 72)])
def test_step_block_is_the_step_of_a_stack(M, D, H):
    """Four launches with sums in an order of their own: the state to fp32 rounding, what lies behind bfloat16
    intermediates to theirs."""
    lib, C = _lib.load(), D // 2
    torch.manual_seed(M + D)

    def bf16(*shape):
        return (torch.randn(shape, device="cuda") / shape[-1] ** 0.5).bfloat16()

    w = dict(in_w=bf16(5 * C, D), out_w16=bf16(D, 2 * D), w12_w=bf16(lib.fields_step_w12_rows(H), D), w3_16=bf16(D, H),
             in_b=torch.randn(5 * C, device="cuda"), par=torch.rand(3, C, device="cuda"), out_b=torch.randn(D, device="cuda"))
    x0, state0 = torch.randn(M, D, device="cuda"), torch.randn(M, D, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def run(call):
        t = dict(w, x=x0, state=state0.clone(), y=torch.empty_like(x0), xb=x0.bfloat16(), yb=bf16(M, D), read=bf16(M, 2 * D),
                 gate=bf16(M, D), act=bf16(M, H), read_sq=torch.empty(C // 8, M, device="cuda"),
                 y_sq=torch.empty(D // 8, M, device="cuda"))
        args = StepArgs(*[t[n].data_ptr() for n, _ in StepArgs._fields_[:17]], 1e-6, 1e-5, M, D, H, 0)
        assert call(ctypes.byref(args)) == 0
        torch.cuda.synchronize()
        return t

    got = run(lambda a: lib.fields_step_block(a, stream))
    want = run(lambda a: lib.fields_step_stack(a, 1, None, stream))
    # fp32 sums of 2,048 products at most err by 2,048 2^-24 of their absolute sum at the very most. Two roundings to bfloat16
    # of nearly the same value are at most neighbours, 2^-7 of it apart; act and y are computed from such values.
    for name, bound in (("state", 2 ** -13), ("read", 2 ** -7), ("gate", 2 ** -7), ("yb", 2 ** -7), ("act", 2 ** -6), ("y", 2 ** -7),
                        ("xb", 2 ** -6)):
        assert torch.isfinite(want[name]).all()
        err = float((got[name].float() - want[name].float()).abs().max())
        assert err <= bound * float(want[name].float().abs().max()), name
