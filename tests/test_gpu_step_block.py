"""fields_step_block through the C ABI, directly behind the layouts that it needs (GPU)."""
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
