"""Retention and the gated delta rule over long portions of prompts in chunks (csrc/linear_chunked.cu) against the recurrence in 64 bits."""

from __future__ import annotations

import math
from types import SimpleNamespace

import pytest
import torch

DEV = torch.device("cuda")


def _operands(lens, H, G, D, V, gated, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    N, cols = sum(lens), 2 * G * D + H * V + (2 * H if gated else 0)
    rec = rnd(N, -(-(cols + G) // 4) * 4)
    qk = rec[:, : 2 * G * D].view(N, 2 * G, D)
    qk /= qk.norm(dim=-1, keepdim=True)
    if gated:
        gates = rec[:, 2 * G * D + H * V:]
        gates[:, :H] = torch.exp(-3 * torch.rand(N, H, generator=g, device=DEV) ** 4)
        gates[:, H // 2: H] *= (torch.rand(N, H - H // 2, generator=g, device=DEV) > 0.02)  # some decays are zero: the state is forgotten
        gates[:, H: 2 * H] = torch.sigmoid(rnd(N, H))
    rec[:, cols: cols + G] = (qk[:, :G] * qk[:, G:]).sum(-1)
    decay = torch.tensor([1.0 - 2.0 ** -(5 + h % 8) for h in range(H)], device=DEV)
    return rec, decay, 0.3 * rnd(len(lens) + 1, H * D * V + 4)


def _walk(rec, decay, state, lens, slots, H, G, D, V, gated):
    outs, after, at = [], state.double().clone(), 0
    for slot, n in zip(slots, lens):
        x = rec[at: at + n].double()
        at += n
        q, k = (x[:, i * G * D: (i + 1) * G * D].view(n, G, D).repeat_interleave(H // G, dim=1) for i in (0, 1))
        v, gates = x[:, 2 * G * D: 2 * G * D + H * V].view(n, H, V), x[:, 2 * G * D + H * V:]
        S = after[slot, : H * D * V].view(H, D, V).clone()
        for t in range(n):
            S = (gates[t, :H] if gated else decay.double())[:, None, None] * S
            u = gates[t, H: 2 * H, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0]) if gated else v[t]
            S = S + k[t][:, :, None] * u[:, None]
            outs.append(torch.bmm(q[t][:, None], S).reshape(-1))
        after[slot, : H * D * V] = S.reshape(-1)
    return torch.stack(outs), after


def _context(lens, slots, ws):
    return SimpleNamespace(n_requests=len(lens), extras={}, q_lens=lens, max_q_len=max(lens), state_slot=torch.tensor(slots, dtype=torch.int32, device=DEV),
                           qo_indptr=torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV),
                           buffer=lambda name, cols, dtype, rows: ws.get(name, rows, cols, dtype))


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("lens,H,G,D,V", [([64], 1, 1, 128, 128), ([65, 3, 129], 4, 2, 128, 128), ([63, 1, 200], 2, 2, 64, 64),
                                          ([130, 66], 6, 2, 64, 192), ([257], 2, 1, 128, 256)])
def test_chunked_recurrence(lens, H, G, D, V, gated, monkeypatch):
    """Requests below and above the chunked walk's least length, remainders of one token to whole chunks, slots in another order than the
    requests.  Bound: every sum has at most 256 + 64 terms, whose roundings (2^-24 each) add up like sqrt(n) in the 2-norm, through about
    four products one after another; a decay of zero stays a number."""
    from nanospec_b200 import ops
    from nanospec_b200.parts import Workspace
    if not gated:
        G = H
    monkeypatch.setattr(ops, "LINEAR_CHUNKED_MIN", 64)
    monkeypatch.setattr(ops, "LINEAR_CHUNKED_COST", (0, 0.0))
    rec, decay, state = _operands(lens, H, G, D, V, gated, sum(lens) + H)
    slots = [len(lens) - i for i in range(len(lens))]
    want, after = _walk(rec, decay, state, lens, slots, H, G, D, V, gated)
    ctx = _context(lens, slots, Workspace(DEV))
    one = 4 * sum(-(-n // 64) for n in lens if n >= 64) * (V * D + 68 + (64 * (D + V) if gated else 0))  # bytes of a head's chunks
    names, call = [], ops.lib.call
    monkeypatch.setattr(ops.lib, "call", lambda name, *a: (names.append(name), call(name, *a)))
    for limit, passes in ((1 << 28, 1), (one, H)):  # all heads in one pass, and a head at a time
        monkeypatch.setattr(ops, "LINEAR_SCRATCH_MAX", limit)
        names.clear()
        S, out = state.clone(), torch.full((sum(lens), H * V + 4), 7.0, device=DEV)
        ops.linear_mix(rec, S, ctx, out[:, : H * V], H, G, D, V, decay=None if gated else decay, gated=gated)
        assert names.count("ns_linear_chunked") == passes and names.count("ns_linear_scan") == (min(lens) < 64)
        bound = 4 * 320 ** 0.5 * 2.0 ** -24
        assert float((out[:, : H * V].double() - want).norm() / want.norm()) < bound
        assert float((S.double() - after).norm() / after.norm()) < bound
        assert bool((out[:, H * V:] == 7.0).all()) and torch.equal(S[0], state[0]) and torch.equal(S[:, H * D * V:], state[:, H * D * V:])


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("H,G,D,V", [(2, 1, 128, 128), (4, 2, 64, 192)])
@pytest.mark.parametrize("bad", [0, 1, 15, 70, 77, 127, 149])
def test_a_token_that_is_no_number_leaves_earlier_ones_alone(bad, H, G, D, V, gated, monkeypatch):
    """A NaN or an infinity in one operand of token `bad` of the first request: everything before it, the other request and the heads and
    columns that it does not enter keep their bits; what the recurrence makes non-finite is non-finite."""
    from nanospec_b200 import ops
    from nanospec_b200.parts import Workspace
    if not gated:
        G = H
    lens, slots = [150, 70], [1, 2]
    monkeypatch.setattr(ops, "LINEAR_CHUNKED_MIN", 64)
    monkeypatch.setattr(ops, "LINEAR_CHUNKED_COST", (0, 0.0))
    rec, decay, state = _operands(lens, H, G, D, V, gated, bad + H)
    ctx = _context(lens, slots, Workspace(DEV))

    def run(r):
        S, out = state.clone(), torch.empty(sum(lens), H * V, device=DEV)
        ops.linear_mix(r, S, ctx, out, H, G, D, V, decay=None if gated else decay, gated=gated)
        return out, S
    clean, S_clean = run(rec)
    v0 = 2 * G * D
    for col, value in [(v0 + V + 5, math.nan), (v0 + V + 5, math.inf), (G * D + 3, math.nan), (G * D + 3, -math.inf), (3, math.nan)] \
            + ([(v0 + H * V + H, math.nan)] if gated else []):
        worse = rec.clone()
        worse[bad, col] = value
        out, S = run(worse)
        want, after = _walk(worse, decay, state, lens, slots, H, G, D, V, gated)
        untouched = torch.ones_like(out, dtype=torch.bool)
        if col >= v0 + H * V:
            untouched[bad: 150, :V] = False                      # the first head's write strength
        elif col >= v0:
            untouched[bad: 150, V + 5] = False                   # one column of the second head's values
        else:
            untouched[bad: 150, : H // G * V] = False            # the first key head
        assert torch.equal(out[untouched], clean[untouched]), (col, value)
        assert not bool(out[~want.isfinite()].isfinite().any()) and not bool(S[~after.isfinite()].isfinite().any()), (col, value)
        assert torch.equal(S[2], S_clean[2])


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [True, False])
def test_a_decay_that_is_no_number_is_carried_on(gated, monkeypatch):
    """A NaN among the decays enters everything from its token (retention: of its head) on, and a decay of zero next to it stays a number."""
    from nanospec_b200 import ops
    from nanospec_b200.parts import Workspace
    H, D, V, lens = 2, 64, 64, [150]
    monkeypatch.setattr(ops, "LINEAR_CHUNKED_MIN", 64)
    monkeypatch.setattr(ops, "LINEAR_CHUNKED_COST", (0, 0.0))
    rec, decay, state = _operands(lens, H, H, D, V, gated, 3)
    at = 2 * H * D + H * V
    if gated:
        rec[60, at: at + 2] = 0.0
        rec[77, at + 1] = math.nan
    else:
        decay[:] = torch.tensor([0.0, math.nan])
    S, out = state.clone(), torch.empty(150, H * V, device=DEV)
    ops.linear_mix(rec, S, _context(lens, [1], Workspace(DEV)), out, H, H, D, V, decay=None if gated else decay, gated=gated)
    want, after = _walk(rec, decay, state, lens, [1], H, H, D, V, gated)
    assert torch.equal(out.isfinite(), want.isfinite()) and torch.equal(S.isfinite(), after.isfinite())
    sound = want.isfinite()
    assert float((out[sound].double() - want[sound]).norm() / want[sound].norm()) < 4 * 320 ** 0.5 * 2.0 ** -24


@pytest.mark.gpu
def test_negative_decays_are_walked():
    """The sign of a fixed decay alternates from token to token, which a sum of logarithms does not hold: such a layer goes token by token."""
    from nanospec_b200 import ops
    from nanospec_b200.config import PartSpec
    from nanospec_b200.parts import Workspace, build_part
    spec = {"hidden": 128, "heads": 2, "head_dim": 64, "v_dim": 64, "eps": 1e-6, "position": None}
    for decay, mix in (((0.5, -0.25), ops.linear_scan), ((0.5, 0.0), ops.linear_mix), ((math.nan, 0.5), ops.linear_scan)):
        part = build_part("mixer", PartSpec("retention", {**spec, "decay": decay}), torch.float32, DEV)
        assert part.mix is mix
    rec, _, state = _operands([300], 2, 2, 64, 64, False, 1)
    decay = torch.tensor([0.9, -0.95], device=DEV)
    part = build_part("mixer", PartSpec("retention", {**spec, "decay": decay.tolist()}), torch.float32, DEV)
    S, out = state.clone(), torch.empty(300, 128, device=DEV)
    part.mix(rec, S, _context([300], [1], Workspace(DEV)), out, 2, 2, 64, 64, decay=decay)
    want, _ = _walk(rec, decay, state, [300], [1], 2, 2, 64, 64, False)
    assert float((out.double() - want).norm() / want.norm()) < 4 * 320 ** 0.5 * 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("H,G,limit,calls", [(6, 1, 6, 1), (6, 1, 4, 2), (6, 1, 1, 6), (6, 2, 5, 2), (6, 2, 2, 4), (6, 2, 0, 0)])
def test_chunk_scratch_stays_below_its_limit(H, G, limit, calls, monkeypatch):
    """Several heads to a key head: passes of parts of one, no more bytes than the limit, the same bits, and the walk where not even one
    head's chunks fit."""
    from nanospec_b200 import ops
    from nanospec_b200.parts import Workspace
    D = V = 64
    lens, one = [200], 4 * 4 * (V * D + 68 + 64 * (D + V))
    monkeypatch.setattr(ops, "LINEAR_CHUNKED_COST", (0, 0.0))
    rec, _, state = _operands(lens, H, G, D, V, True, 7)
    names, call = [], ops.lib.call
    monkeypatch.setattr(ops.lib, "call", lambda name, *a: (names.append(name), call(name, *a)))
    outs = []
    for most in (1 << 28, limit * one + 15):
        monkeypatch.setattr(ops, "LINEAR_SCRATCH_MAX", most)
        names.clear()
        ws, S, out = Workspace(DEV), state.clone(), torch.empty(200, H * V, device=DEV)
        ops.linear_mix(rec, S, _context(lens, [1], ws), out, H, G, D, V, gated=True)
        outs.append((out, S))
        assert sum(b.numel() * b.element_size() for b in ws._bufs.values()) <= most + 32
    assert names == ["ns_linear_chunked"] * calls or (not calls and names == ["ns_linear_scan"])
    if calls:
        assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("lens,H,D,V,gated,chunked", [
    # us by token, in chunks (B200)
    ([1000], 16, 128, 128, True, True),              # 304, 134
    ([256], 32, 128, 128, True, True),               # 106, 90
    ([600, 100], 16, 128, 128, True, True),          # 228, 143
    ([2048, 2048], 16, 128, 128, True, True),        # 818, 538
    ([2000] + [1] * 7, 32, 128, 128, True, True),    # 1056, 540
    ([300] * 4, 4, 64, 64, True, True),              # 77, 51
    ([300] * 4, 16, 128, 128, False, True),          # 153, 103
    ([192, 191], 16, 128, 128, True, False),         # 81, 147
    ([300, 150], 16, 128, 128, True, False),         # 120, 142
    ([300] * 4, 16, 128, 128, True, False),          # 171, 199
    ([2048, 2048], 32, 128, 128, True, False),       # 1134, 1184
    ([300] * 4, 16, 64, 64, True, False),            # 88, 106
    ([1000] * 8, 16, 64, 64, True, False),           # 413, 545
    ([300] * 16, 4, 64, 64, True, False),            # 89, 107
    ([192, 191], 4, 64, 64, False, False),           # 47, 69
    ([191], 4, 64, 64, False, False), ([2048], 16, 256, 64, True, False), ([], 16, 64, 64, True, False),
])
def test_chunks_are_taken_where_they_are_faster(lens, H, D, V, gated, chunked, monkeypatch):
    from nanospec_b200 import ops
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    assert ops.chunks_pay(lens, H, D, V, gated) == chunked


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("others,chunked", [([], True), ([1], True), ([190], False), ([300] * 7, False)])
def test_a_long_request_beside_others(others, chunked, gated, monkeypatch):
    """The rule as it stands, on both its sides: a request's numbers depend on its neighbours by the roundings of its sums alone (the walk and the
    chunks each within the bound of `test_chunked_recurrence` of the recurrence in 64 bits)."""
    from nanospec_b200 import ops
    from nanospec_b200.parts import Workspace
    H, G, D, V = 16, 8 if gated else 16, 128, 128
    lens = [300, *others]
    names, call = [], ops.lib.call
    monkeypatch.setattr(ops.lib, "call", lambda name, *a: (names.append(name), call(name, *a)))
    rec, decay, state = _operands(lens, H, G, D, V, gated, len(others))
    want, after = _walk(rec[:300], decay, state, [300], [1], H, G, D, V, gated)
    S, out = state.clone(), torch.empty(sum(lens), H * V, device=DEV)
    ops.linear_mix(rec, S, _context(lens, [i + 1 for i in range(len(lens))], Workspace(DEV)), out, H, G, D, V, decay=None if gated else decay, gated=gated)
    assert ("ns_linear_chunked" in names) == chunked
    bound = 4 * 320 ** 0.5 * 2.0 ** -24
    assert float((out[:300].double() - want).norm() / want.norm()) < bound
    assert float((S[1].double() - after[1]).norm() / after[1].norm()) < bound
