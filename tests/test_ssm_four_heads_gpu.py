"""The chunked state space with four heads to a block against the kernels that take a head alone, bit for bit."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("lens,H,G", [([96], 4, 1), ([97, 3, 191], 8, 2), ([128, 65, 160], 12, 1), ([511], 16, 4), ([577, 1153], 4, 1)])
def test_four_heads_to_a_block(lens, H, G, N, monkeypatch):
    from nanospec_b200 import ops
    monkeypatch.setattr(ops, "SSM_FOUR_HEADS_FROM", 0)  # also where they are too few to be worth it
    from nanospec_b200.parts import Workspace
    V = 64
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + H + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    T, off, per = sum(lens), 2 * G * N, H // G
    rec = rnd(T, -(-(off + H * V + 2 * H + G) // 4) * 4)
    a_log, step = 0.5 * rnd(H), torch.nn.functional.softplus(rnd(T, H))
    step[:, 0] *= 30  # a head that forgets at once
    rec[:, off + H * V: off + H * V + H] = torch.exp(-torch.exp(a_log) * step)
    rec[:, off + H * V + H: off + H * V + 2 * H] = step
    rec[:, off + H * V + 2 * H: off + H * V + 2 * H + G] = (rec[:, : G * N] * rec[:, G * N: off]).view(T, G, N).sum(-1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    ws = Workspace(DEV)
    ctx = SimpleNamespace(n_requests=len(lens), extras={}, q_lens=lens, max_q_len=max(lens), state_slot=i32([len(lens) - i for i in range(len(lens))]),
                          qo_indptr=i32([sum(lens[:i]) for i in range(len(lens) + 1)]), buffer=lambda name, cols, dtype, rows: ws.get(name, rows, cols, dtype))
    state = 0.3 * rnd(len(lens) + 1, H * N * V)
    S, out = state.clone(), torch.full((T, H * V + 4), 7.0, device=DEV)
    ops.ssm_scan(rec, a_log, S, ctx, out[:, : H * V], H, G, N, V)
    for h in range(H):
        q = h // per
        one = torch.cat([rec[:, q * N: (q + 1) * N], rec[:, (G + q) * N: (G + q + 1) * N], rec[:, off + h * V: off + (h + 1) * V],
                         rec[:, off + H * V + h, None], rec[:, off + H * V + H + h, None], rec[:, off + H * V + 2 * H + q, None], rec[:, :1]], dim=1).contiguous()
        S1, o1 = state[:, h * N * V: (h + 1) * N * V].contiguous(), torch.empty(T, V, device=DEV)
        ops.ssm_scan(one, a_log[h: h + 1].clone(), S1, ctx, o1, 1, 1, N, V)
        assert torch.equal(out[:, h * V: (h + 1) * V], o1), h
        assert torch.equal(S[:, h * N * V: (h + 1) * N * V], S1), h
    assert bool((out[:, H * V:] == 7.0).all())


@pytest.mark.parametrize("tokens,heads,blocks", [(96, 32, 16), (500, 64, 128), (300, 128, 160)])
def test_both_sides_of_the_rule_give_the_same_bits(tokens, heads, blocks, monkeypatch):
    """A step below and above the number of SMs in blocks of four heads, as the rule has it and with the other choice."""
    from nanospec_b200 import ops
    from nanospec_b200.parts import Workspace
    assert -(-tokens // 64) * heads // 4 == blocks
    N, V, G = 64, 64, 8
    g = torch.Generator(device=DEV).manual_seed(tokens)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    off = 2 * G * N + heads * V
    rec, a_log, step = rnd(tokens, off + 2 * heads + G), 0.5 * rnd(heads), torch.nn.functional.softplus(rnd(tokens, heads))
    rec[:, off: off + heads], rec[:, off + heads: off + 2 * heads] = torch.exp(-torch.exp(a_log) * step), step
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    ws, state = Workspace(DEV), 0.3 * rnd(2, heads * N * V)
    ctx = SimpleNamespace(n_requests=1, extras={}, q_lens=[tokens], max_q_len=tokens, state_slot=i32([1]), qo_indptr=i32([0, tokens]),
                          buffer=lambda name, cols, dtype, rows: ws.get(name, rows, cols, dtype))
    seen, call = [], ops.lib.call
    monkeypatch.setattr(ops.lib, "call", lambda name, *a: (seen.append((name, a[-2])), call(name, *a)))
    outs = []
    for least in (None, 0, 1 << 20):
        monkeypatch.setattr(ops, "SSM_FOUR_HEADS_FROM", least)
        S, out = state.clone(), torch.empty(tokens, heads * V, device=DEV)
        ops.ssm_scan(rec, a_log, S, ctx, out, heads, G, N, V)
        outs.append((out, S))
    assert seen == [("ns_ssm_chunked", ops.sm_count()), ("ns_ssm_chunked", 0), ("ns_ssm_chunked", 1 << 20)]
    assert all(torch.equal(a, b) for other in outs[1:] for a, b in zip(outs[0], other))
