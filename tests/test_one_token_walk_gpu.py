"""The recurrences' kernel for steps of one token a request against the kernel that walks tokens, bit for bit."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("kind", ["plain", "delta", "step"])
@pytest.mark.parametrize("B,H,G,D,V", [(1, 1, 1, 16, 64), (5, 6, 3, 32, 64), (3, 4, 2, 64, 192), (17, 8, 8, 128, 128), (2, 3, 3, 256, 64)])
def test_one_token_a_request(kind, B, H, G, D, V):
    from nanospec_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(B + D + V)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    gated = kind != "plain"
    if not gated:
        G = H
    off = 2 * G * D + H * V
    rec = rnd(B, -(-(off + 2 * H + G) // 4) * 4)
    rec[:, off: off + 2 * H].sigmoid_()
    decay, state = torch.rand(H, generator=g, device=DEV), rnd(B + 1, H * D * V + 4)
    lens = [1] * B
    if B > 2:
        lens[1] = 0  # a request that brings nothing keeps its state
    ctx = SimpleNamespace(n_requests=B, max_q_len=1, qo_indptr=torch.tensor([sum(lens[:i]) for i in range(B + 1)], dtype=torch.int32, device=DEV),
                          state_slot=torch.randperm(B + 1, generator=torch.Generator().manual_seed(1))[:B].int().to(DEV))
    got = []
    for longest in (1, 2):  # (2: the walk)
        S, out = state.clone(), torch.full((B, H * V + 3), 7.0, device=DEV)
        ops.linear_scan(rec, S, ctx, out[:, : H * V], H, G, D, V, decay=None if gated else decay, gated=gated, delta=kind == "delta", longest=longest)
        got.append((S, out))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert not torch.equal(got[0][0], state) and torch.equal(got[0][0][:, H * D * V:], state[:, H * D * V:])
