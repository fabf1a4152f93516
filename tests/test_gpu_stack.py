"""The native inference path of FieldStackDecoder (csrc/torch_stack.cpp, field_rows.cuh) against the
same decoder running the model's modules one by one (GPU)."""
import pytest
import torch

import mirror
from conftest import BF16_TOL
from fields_lm_b200 import FieldStackDecoder, stack

pytestmark = pytest.mark.gpu


class LM(torch.nn.Module):
    def __init__(self, dim, layers, hidden, bias=False):
        super().__init__()
        self.emb = torch.nn.Embedding(97, dim)
        self.blocks = torch.nn.ModuleList(mirror.FieldBlock(dim, ff_hidden=hidden) for _ in range(layers))
        self.final_norm = mirror.RMSNorm(dim)
        self.lm_head = torch.nn.Linear(dim, 97, bias=bias)


def _rel(a, b):
    return float((a.float() - b.float()).abs().max() / b.float().abs().max().clamp_min(1e-6))


def _run(model, tokens, prefix, native):
    dec = FieldStackDecoder(model)
    dec._refused = not native
    plan = stack.plan
    if not native:
        stack.plan = lambda *a: None
    try:
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = [dec.prefill(tokens[:, :prefix], last_only=False)[:, -1]]
            out += [dec.step(tokens[:, t]) for t in range(prefix, tokens.shape[1])]
    finally:
        stack.plan = plan
    assert (dec._stack is not None) == native
    return out, dec


# one block's rounding differences grow by at most their sum over the blocks: BF16_TOL holds for three
# (fused step: rows around one tile of 128 and its limit of 512, widths that leave part of a column
# tile, K shorter than the split; 200 and 1032 are widths it does not take)
@pytest.mark.parametrize("dim,hidden,B,L", [(64, 8, 1, 1), (64, 40, 5, 3), (200, 96, 3, 37), (1024, 2528, 2, 64),
                                            (1024, 704, 601, 8), (1032, 352, 4, 5), (4096, 64, 2, 6),
                                            (1024, 2528, 129, 2), (512, 1344, 512, 2), (16, 24, 127, 2),
                                            (272, 360, 128, 3), (256, 704, 256, 2)])
def test_native_stack_matches_the_modules(dim, hidden, B, L):
    torch.manual_seed(dim + B)
    model = LM(dim, 3, hidden, bias=dim == 200).cuda()
    for p in model.parameters():  # norm weights away from one
        if p.dim() == 1 and p.numel() in (dim, 2 * dim):
            p.data += 0.1 * torch.randn_like(p)
    tokens = torch.randint(0, 97, (B, L + 3), device="cuda")
    got, dec = _run(model, tokens, L, True)
    want, ref = _run(model, tokens, L, False)
    for a, b in zip(got, want):
        assert a.shape == b.shape and a.dtype == b.dtype
        assert _rel(a, b) < BF16_TOL
    for a, b in zip(dec.states, ref.states):
        assert a.dtype == torch.float32 and _rel(a, b) < BF16_TOL


# where one launch and four, fused and library products take turns: rows and tiles of steps, rows of prefills
@pytest.mark.parametrize("dim,hidden,B,L", [(64, 40, 65, 2), (64, 40, 257, 2), (80, 24, 128, 2), (1024, 704, 512, 2), (1280, 64, 384, 4),
                                            (1280, 64, 385, 4), (2048, 96, 256, 2), (2560, 64, 64, 3), (2560, 64, 65, 3),
                                            (768, 352, 3, 5), (1024, 704, 4, 384), (768, 352, 3, 256), (768, 352, 1, 769), (768, 352, 3, 512),
                                            (704, 352, 4, 193), (712, 360, 4, 192), (712, 360, 1, 769)])
def test_edges_of_the_rules(dim, hidden, B, L):
    test_native_stack_matches_the_modules(dim, hidden, B, L)


def test_step_on_states_that_are_not_aligned():
    torch.manual_seed(2)
    model = LM(64, 2, 32).cuda()
    tokens = torch.randint(0, 97, (3, 6), device="cuda")
    _, dec = _run(model, tokens, 6, True)
    odd = []
    for s in dec.states:
        odd.append(torch.zeros(s.numel() + 1, device="cuda")[1:].view_as(s).copy_(s))
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = dec.step(tokens[:, 0])
        after, dec.states = dec.states, odd
        assert torch.equal(dec.step(tokens[:, 0]), want)
    assert all(torch.equal(a, b) for a, b in zip(after, odd))


def test_native_stack_follows_the_model():
    """Weights written in place, replaced or hooked after the prefill are seen by the next step."""
    torch.manual_seed(0)
    model = LM(64, 2, 32).cuda()
    tokens = torch.randint(0, 97, (4, 6), device="cuda")
    _, dec = _run(model, tokens, 6, True)

    def step():
        states = [s.clone() for s in dec.states]
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = dec.step(tokens[:, 0])
        dec.states = states
        return out

    before = step()
    assert torch.equal(before, step())
    with torch.no_grad():
        model.blocks[1].ff.w3.weight.mul_(3.0)
    changed = step()
    assert _rel(changed, before) > BF16_TOL
    with torch.no_grad():
        model.blocks[1].ff.w3.weight.div_(3.0)
    assert _rel(step(), before) < BF16_TOL
    model.blocks[1].ff.w3.weight = torch.nn.Parameter(model.blocks[1].ff.w3.weight.detach() * 3.0)
    assert _rel(step(), changed) < BF16_TOL
    seen = []
    model.blocks[0].ff_norm.register_forward_hook(lambda *a: seen.append(1))
    assert _rel(step(), changed) < BF16_TOL and seen and dec._stack is None


def test_model_of_inference_tensors():
    """Parameters that have no version counter: the weights as they are at every step."""
    torch.manual_seed(1)
    plain = LM(64, 2, 32).cuda()
    with torch.inference_mode():
        model = LM(64, 2, 32).cuda()
        model.load_state_dict(plain.state_dict())
    assert all(p.is_inference() for p in model.parameters())
    tokens = torch.randint(0, 97, (4, 8), device="cuda")
    got, want = _run(model, tokens, 5, True), _run(plain, tokens, 5, True)
    assert all(torch.equal(a, b) for a, b in zip(got[0], want[0]))
    for m in (model, plain):
        with torch.inference_mode():
            m.blocks[1].ff.w3.weight.mul_(3.0)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert torch.equal(got[1].step(tokens[:, 0]), want[1].step(tokens[:, 0]))
        assert torch.equal(got[1].prefill(tokens), want[1].prefill(tokens))


def test_captured_step_and_prefill_follow_the_weights():
    """A graph replays with the weights of that moment, and does not need the decoder it was captured from."""
    torch.manual_seed(3)
    model = LM(64, 2, 32).cuda()
    tokens = torch.randint(0, 97, (4, 6), device="cuda")
    _, dec = _run(model, tokens, 6, True)
    kept = [s.clone() for s in dec.states]

    def eager():
        ref = FieldStackDecoder(model)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            first = ref.prefill(tokens)
            ref.states = [s.clone() for s in kept]
            return ref.step(tokens[:, 0]), first

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        eager()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), torch.cuda.graph(graph, stream=side):
        states, dec.states = dec.states, [s.clone() for s in dec.states]
        out = dec.step(tokens[:, 0])
        first = dec.prefill(tokens)
    dec.states = states
    assert not dec._refused
    with torch.autocast("cuda", dtype=torch.bfloat16):
        dec.prefill(tokens)  # what was captured is no layout of the decoder's own
        assert _rel(dec.step(tokens[:, 0]), eager()[0]) < 1e-6
    dec.reset()
    for factor in (1.0, 3.0, 0.5):
        with torch.no_grad():
            model.blocks[1].ff.w3.weight.mul_(factor)
            model.blocks[0].mixer.gate_proj.bias.add_(factor)
        graph.replay()
        torch.cuda.synchronize()
        for got, want in zip((out, first), eager()):
            assert _rel(got, want) < 1e-6


@pytest.mark.parametrize("width", [32, 128])
def test_activations_of_another_width_are_refused(width):
    torch.manual_seed(4)
    model = LM(64, 2, 32).cuda()
    tokens = torch.randint(0, 97, (3, 6), device="cuda")
    _, dec = _run(model, tokens, 6, True)
    model.emb = torch.nn.Embedding(97, width).cuda()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        with pytest.raises(RuntimeError):
            dec.step(tokens[:, 0])
        with pytest.raises(RuntimeError):
            dec.prefill(tokens)


def test_activations_that_are_not_aligned():
    class Shifted(torch.nn.Embedding):
        def forward(self, tokens):
            x = super().forward(tokens)
            return torch.zeros(x.numel() + 1, device=x.device)[1:].view_as(x).copy_(x)

    torch.manual_seed(5)
    model = LM(64, 2, 32).cuda()
    tokens = torch.randint(0, 97, (3, 8), device="cuda")
    want, _ = _run(model, tokens, 5, True)
    model.emb.__class__ = Shifted
    got, _ = _run(model, tokens, 5, True)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_calls_on_other_streams_wait_for_the_copies():
    """A step on a stream that does not wait for the one of the layout, a layout on one that does not wait for the one
    of a step, and a decoder that goes away while its last call is pending."""
    torch.manual_seed(6)
    model = LM(256, 4, 704).cuda()
    tokens = torch.randint(0, 97, (8, 12), device="cuda")
    _, ref = _run(model, tokens, 12, True)
    kept = [s.clone() for s in ref.states]
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = ref.step(tokens[:, 0])
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        dec = FieldStackDecoder(model)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            dec._native_stack(model.emb(tokens))  # (making the plan waits for the GPU)
            states = [s.clone() for s in kept]
            torch.cuda.synchronize()
            with torch.cuda.stream(a):
                torch.cuda._sleep(20_000_000)
                dec.prefill(tokens)
            dec.states = states
            with torch.cuda.stream(b):
                got = dec.step(tokens[:, 0])
            with torch.cuda.stream(a):
                torch.cuda._sleep(20_000_000)
                dec.states = [s.clone() for s in kept]
                again = dec.step(tokens[:, 0])
            with torch.cuda.stream(b):
                other = dec.prefill(tokens)
                dec.states = None
            del dec
            with torch.cuda.stream(a):
                junk = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(64)]
        torch.cuda.synchronize()
        assert torch.equal(got, want) and torch.equal(again, want) and not bool(other.isnan().any())
        del junk


# (rows of the first call and of the late one, which needs weights in another order: the fused step, the step with library
# products, the prefill with fused products behind one with library products and the other way round)
@pytest.mark.parametrize("dim,hidden,B,first,late", [(256, 704, 8, 12, "step"), (64, 40, 513, 2, "step"), (1024, 704, 2, 3, 1024),
                                                     (1024, 704, 2, 1024, 3)])
def test_copies_made_on_the_way_outlive_their_calls(dim, hidden, B, first, late):
    """Copies that a call on b was the first to need are read by a pending call on a when the decoder goes away; what b
    allocates next does not get their memory before that call is done."""
    torch.manual_seed(8)
    model = LM(dim, 2, hidden).cuda()
    tokens = torch.randint(0, 97, (B, 1024 if dim == 1024 else 12), device="cuda")
    kept = [torch.randn(B, dim, device="cuda") for _ in model.blocks]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()

    def call(dec):
        if late != "step":
            return dec.prefill(tokens[:, :late])
        dec.states = [s.clone() for s in kept]
        return dec.step(tokens[:, 0])

    with torch.autocast("cuda", dtype=torch.bfloat16):
        ref = FieldStackDecoder(model)
        ref.prefill(tokens[:, :first])
        want = call(ref)
        for _ in range(3):
            dec = FieldStackDecoder(model)
            dec._native_stack(model.emb(tokens))
            torch.cuda.synchronize()
            with torch.cuda.stream(a):
                dec.prefill(tokens[:, :first])
            torch.cuda.synchronize()
            with torch.cuda.stream(b):
                call(dec)
            torch.cuda.synchronize()
            with torch.cuda.stream(a):
                torch.cuda._sleep(20_000_000)
                got = call(dec)
            del dec
            with torch.cuda.stream(b):  # (of the sizes of the copies)
                junk = [torch.full((rows, dim), float("nan"), device="cuda", dtype=torch.bfloat16)
                        for rows in (2 * hidden, (hidden + 19) // 20 * 40, 5 * dim // 2) for _ in range(8)]
            torch.cuda.synchronize()
            assert torch.equal(got, want)
            del junk


def test_first_step_leaves_the_w12_of_the_prefill():
    """A prefill with fused products has laid out w12 in the order of the step: the step does not write it again (a call on
    another stream may be reading it), so a write that torch does not count is not seen."""
    torch.manual_seed(9)
    model = LM(64, 2, 40).cuda()
    tokens = torch.randint(0, 97, (3, 6), device="cuda")
    _, ref = _run(model, tokens, 6, True)
    _, dec = _run(model, tokens, 6, True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = ref.step(tokens[:, 0])
        for b in model.blocks:
            b.ff.w12.weight.data.mul_(-3.0)
        assert torch.equal(dec.step(tokens[:, 0]), want)


def test_library_step_uses_the_weights_of_the_prefill():
    """... and so does the step with library products behind a prefill with fused ones."""
    torch.manual_seed(10)
    model = LM(64, 2, 40).cuda()
    tokens = torch.randint(0, 97, (513, 3), device="cuda")
    _, ref = _run(model, tokens, 3, True)
    _, dec = _run(model, tokens, 3, True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = ref.step(tokens[:, 0])
        for b in model.blocks:
            b.ff.w12.weight.data.mul_(-3.0)
        assert torch.equal(dec.step(tokens[:, 0]), want)


# (the step as four launches per block, as one, and with library products)
@pytest.mark.parametrize("dim,B", [(64, 3), (384, 3), (64, 520)])
def test_nan_stays_in_its_sequence(dim, B):
    """A NaN embedding: NaN logits from that token on in its sequence and nowhere else, through the prefill and a step; so
    does a NaN in a state."""
    torch.manual_seed(11)
    model = LM(dim, 2, 40).cuda()
    with torch.no_grad():
        model.emb.weight[5] = float("nan")
    tokens = torch.randint(6, 97, (B, 9), device="cuda")
    tokens[1, 4] = 5
    dec = FieldStackDecoder(model)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        logits = dec.prefill(tokens, last_only=False)
        assert dec._stack is not None
        bad = logits.isnan()
        assert bool(bad[1, 4:].all()) and int(bad.sum()) == bad[1, 4:].numel()
        dec.states[0][2, 7] = float("nan")
        bad = dec.step(tokens[:, 0]).isnan()
    assert bool(bad[1:3].all()) and int(bad.sum()) == bad[1:3].numel()


def test_threads_share_a_decoder():
    import threading
    torch.manual_seed(7)
    model = LM(128, 3, 352).cuda()
    batches = [torch.randint(0, 97, (4, 9 + i), device="cuda") for i in range(4)]
    want = [_run(model, t, t.shape[1], True)[0][0] for t in batches]
    dec, bad = FieldStackDecoder(model), []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()), torch.autocast("cuda", dtype=torch.bfloat16):
                for _ in range(30):
                    got = dec.prefill(batches[i])
                    torch.cuda.current_stream().synchronize()
                    assert _rel(got, want[i]) < 1e-6
        except BaseException as e:  # noqa: BLE001
            bad.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
