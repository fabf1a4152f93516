"""The one-launch scan kernels (csrc/field_scan.cuh) at the edges of their tiles and clusters, against
the oracle (GPU). A tile is 128 steps of 32 channels, a cluster up to 16 tiles."""
import numpy as np
import pytest
import torch

from conftest import FP32_TOL, rel_err
from fields_lm_b200 import linear_scan_with_state
from oracle import scan_oracle

pytestmark = pytest.mark.gpu


# steps around one thread (16), one tile (128), one cluster (2,048) and several super-tiles; channels
# around one warp; chains from one to more than the GPU holds blocks
@pytest.mark.parametrize("B,L,C", [(1, 1, 1), (2, 15, 31), (2, 17, 33), (1, 127, 32), (3, 129, 64), (1, 2048, 64),
                                   (1, 2049, 64), (2, 4500, 40), (40, 300, 100), (160, 257, 64), (310, 130, 32)])
@pytest.mark.parametrize("shared", [True, False])
def test_scan_walk_matches_the_oracle(B, L, C, shared):
    rng = np.random.default_rng(B * 1000 + L + C)
    a = rng.uniform(0.01, 0.999, (B, L, 1 if shared else C)).astype(np.float32)
    drive, grad = (rng.standard_normal((B, L, C)).astype(np.float32) for _ in range(2))
    first, last = (rng.standard_normal((B, C)).astype(np.float32) for _ in range(2))
    want, want_end = scan_oracle.forward(a, drive, first)
    want_a, want_b, want_first = scan_oracle.backward(a, drive, grad, first, last)
    leaves = [torch.from_numpy(t).cuda().requires_grad_(True) for t in (a, drive, first)]
    states, end = linear_scan_with_state(leaves[0].expand(B, L, C), leaves[1], leaves[2])
    assert torch.equal(end, states[:, -1])
    got = torch.autograd.grad([states, end], leaves, [torch.from_numpy(t).cuda() for t in (grad, last)])
    assert rel_err(states.detach().cpu().numpy(), want) < FP32_TOL
    assert rel_err(end.detach().cpu().numpy(), want_end) < FP32_TOL
    want_a = want_a.sum(axis=2, keepdims=True) if shared else want_a
    for g, w in zip(got, (want_a, want_b, want_first)):
        assert rel_err(g.cpu().numpy(), w) < FP32_TOL
