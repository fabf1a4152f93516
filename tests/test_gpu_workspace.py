"""Passes on the kept workspaces of the torch layer (csrc/torch_api.h): extents and dtypes in any order,
several streams and threads, and graphs, against passes that fill a workspace of their own (GPU)."""
import threading

import numpy as np
import pytest
import torch

from conftest import FP32_TOL, rel_err
from fields_lm_b200 import field_read_with_state, fused_field_read, fused_field_read_bf16
from oracle import field_oracle

pytestmark = pytest.mark.gpu


def _case(B, L, C, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ring, theta = torch.linspace(0.85, 0.999, C, device="cuda"), torch.linspace(0.03, 3.04, C, device="cuda")
    par = [ring * theta.cos(), ring * theta.sin(), (1 - ring ** 2).sqrt()]
    raw = 0.577 * torch.randn(B, L, 3 * C, device="cuda", generator=g)
    return [t.requires_grad_(True) for t in (raw, *par)], torch.randn(B, L, 4 * C, device="cuda", generator=g)


def _pass(leaves, grad):
    read = fused_field_read(*leaves)
    return [read.detach(), *torch.autograd.grad(read, leaves, grad)]


# the fold of the parameter gradients into the last block: one row, the most it takes (16) and one more
@pytest.mark.parametrize("B,L,C", [(1, 1, 4), (2, 250, 132), (16, 32, 260), (17, 31, 128), (1, 513, 512)])
def test_folded_parameter_gradients_match_the_oracle(B, L, C):
    leaves, grad = _case(B, L, C, L)
    host = [t.detach().cpu().numpy() for t in leaves]
    want = [field_oracle.forward(*host)[0], *field_oracle.backward(*host, grad.cpu().numpy())[:4]]
    for _ in range(2):  # the counters are back at their first value
        for g, w in zip(_pass(leaves, grad), want):
            assert rel_err(g.cpu().numpy(), np.asarray(w)) < FP32_TOL


def test_extents_and_forms_in_any_order():
    shapes = [(1, 40, 512), (2, 3001, 384), (3, 777, 132), (1, 300, 7), (1, 40, 512), (8, 512, 512), (1, 1, 4)]
    cases = [_case(*s, i) for i, s in enumerate(shapes)]
    want = [[t.cpu() for t in _pass(*c)] for c in cases]
    for i in [3, 1, 0, 5, 2, 6, 4, 1, 3, 0, 2, 5]:
        leaves, grad = cases[i]
        fused_field_read_bf16(leaves[0].detach().bfloat16(), *[t.detach() for t in leaves[1:]]) if shapes[i][2] % 4 == 0 else None
        field_read_with_state(*leaves, None, lean=True)[0].sum().backward()
        for g, w in zip(_pass(leaves, grad), want[i]):
            assert rel_err(g.cpu().numpy(), w.numpy()) < 1e-6


# the reduction of a backward pass fills both halves: after passes without it (none, one, two, more of them),
# below and above the extent up to which a pass fills for itself, and with halves of unlike extent
@pytest.mark.parametrize("B,L,C", [(17, 31, 132), (2, 1500, 384), (8, 2048, 512)])
def test_halves_after_forwards_alone(B, L, C):
    leaves, grad = _case(B, L, C, 5)
    host = [t.detach().cpu().numpy() for t in leaves]
    want = [field_oracle.forward(*host)[0], *field_oracle.backward(*host, grad.cpu().numpy())[:4]]
    other = [t.detach() for t in _case(3, 1900, 512, 6)[0]]
    for forwards in (0, 1, 2, 3, 0, 0):
        with torch.no_grad():
            for i in range(forwards):
                fused_field_read(*(other if i == 1 else leaves))
        for g, w in zip(_pass(leaves, grad), want):
            assert rel_err(g.cpu().numpy(), np.asarray(w)) < FP32_TOL


def test_streams_and_threads():
    cases = [_case(2, 1500 + 100 * i, 256, i) for i in range(4)]
    want = [[t.cpu() for t in _pass(*c)] for c in cases]
    torch.cuda.synchronize()
    shared = torch.cuda.Stream()
    bad = []

    def work(i):
        stream = shared if i % 2 else torch.cuda.Stream()
        try:
            with torch.cuda.stream(stream):
                for _ in range(20):
                    got = _pass(*cases[i])
                    stream.synchronize()
                    for g, w in zip(got, want[i]):
                        assert rel_err(g.cpu().numpy(), w.numpy()) < 1e-6
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_captured_passes_can_be_replayed():
    leaves, grad = _case(2, 900, 256, 3)
    par = [t.detach() for t in leaves[1:]]
    raw = leaves[0].detach().clone()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side), torch.no_grad():
        fused_field_read(raw, *par)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph, stream=side):
        out = fused_field_read(raw, *par)
    for seed in (11, 12, 13):
        raw.copy_(_case(2, 900, 256, seed)[0][0].detach())
        graph.replay()
        torch.cuda.synchronize()
        got = out.clone()
        with torch.no_grad():
            want = fused_field_read(raw, *par)
        assert rel_err(got.cpu().numpy(), want.cpu().numpy()) < 1e-6


@pytest.mark.parametrize("B,L,C", [(1, 10_000, 33), (2, 3000, 333)])
def test_odd_width_on_a_workspace_of_its_own(B, L, C):
    """Passes whose slots take more than the least half, on a stream that has kept none yet."""
    leaves, grad = _case(B, L, C, 7)
    host = [t.detach().cpu().numpy() for t in leaves]
    want = [field_oracle.forward(*host)[0], *field_oracle.backward(*host, grad.cpu().numpy())[:4]]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        got = _pass(leaves, grad)
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert rel_err(g.cpu().numpy(), np.asarray(w)) < FP32_TOL


def _limit(room):
    """Lets this process reserve `room` more bytes than it has."""
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room) / total)


def _take_back():
    """Leaves no workspace kept by earlier passes."""
    torch.cuda.synchronize()
    try:
        _limit(0)
        with pytest.raises(torch.cuda.OutOfMemoryError):
            torch.empty(8 << 30, dtype=torch.uint8, device="cuda")
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    torch.cuda.empty_cache()


def test_a_failed_allocation_leaves_nothing_behind():
    """A pass without memory for a kept workspace (96 MiB here) but for its own (28 MB), one without memory for
    either, then one on a workspace of its own (above the most that is kept) and the first one again."""
    few, many = _case(1, 300_000, 4, 1), _case(1, 360_000, 4, 2)
    par = [t.detach() for t in few[0][1:]]
    small, large = few[0][0].detach(), many[0][0].detach()
    host = [p.cpu().numpy() for p in par]
    want = {id(t): field_oracle.forward(t.cpu().numpy(), *host)[0] for t in (small, large)}
    stream = torch.cuda.Stream()
    _take_back()
    with torch.cuda.stream(stream):
        try:
            _limit(70 << 20)
            got = [(small, fused_field_read(small, *par).cpu())]
            torch.cuda.empty_cache()
            _limit(30 << 20)
            with pytest.raises(torch.cuda.OutOfMemoryError):
                fused_field_read(small, *par)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        got += [(t, fused_field_read(t, *par).cpu()) for t in (large, small, large, small)]
    for t, g in got:
        assert rel_err(g.numpy(), want[id(t)]) < FP32_TOL


def test_kept_workspaces_are_given_back():
    """What other streams keep is there for an allocation that needs it, and the passes after it are right."""
    leaves, grad = _case(1, 300_000, 4, 3)
    par, raw = [t.detach() for t in leaves[1:]], leaves[0].detach()
    want = torch.from_numpy(field_oracle.forward(raw.cpu().numpy(), *[p.cpu().numpy() for p in par])[0])
    streams = [torch.cuda.Stream() for _ in range(6)]
    _take_back()
    before = torch.cuda.memory_allocated()
    for s in streams:
        with torch.cuda.stream(s):
            fused_field_read(raw, *par)
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated() - before
    assert held > 300 << 20
    torch.cuda.empty_cache()
    try:
        _limit(100 << 20)
        big = torch.empty(held, dtype=torch.uint8, device="cuda")
        del big
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.cuda.memory_allocated() < before + held // 2
    for s in streams:
        with torch.cuda.stream(s):
            assert rel_err(fused_field_read(raw, *par).cpu().numpy(), want.numpy()) < FP32_TOL


@pytest.mark.parametrize("which", range(4))
@pytest.mark.parametrize("grad", [True, False])
def test_forward_mode_tangents_are_refused(which, grad):
    """None of the operators has a forward-mode derivative; a tangent is not dropped in silence."""
    import torch.autograd.forward_ad as fwd
    leaves = [t.detach() for t in _case(1, 20, 8, 1)[0]]
    with fwd.dual_level(), torch.set_grad_enabled(grad):
        leaves[which] = fwd.make_dual(leaves[which], torch.ones_like(leaves[which]))
        with pytest.raises(RuntimeError):
            fused_field_read(*leaves)
        with pytest.raises(RuntimeError):
            field_read_with_state(*leaves)
