"""The chunked state space's read-out on the tensor cores (csrc/ssm_chunked.cu) against the recurrence in 64 bits."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("lens,H,G,four", [([64], 4, 1, 0), ([65, 127], 3, 3, 0), ([96, 79], 8, 2, 0), ([129], 5, 1, 1 << 20), ([200, 2, 113], 4, 2, 1 << 20)])
@pytest.mark.parametrize("speed", [0.1, 1.0, 20.0])
def test_read_out(lens, H, G, four, N, speed, monkeypatch):
    """Full and ragged chunks (one token, one more or less than a tile of 16), one head and four to a block, heads that forget slowly and at once.
    The bound: y is a sum of |decay| |C| |B| |x| products, whose terms pass 24 products' truncations and roundings of 2^-23 each, the states'
    and weights' own roundings (64 sums of 2^-24 and an exponential's 2^-22) among them."""
    _compare(lens, H, G, four, N, speed, monkeypatch)


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("lens,H,G,four", [([96, 79], 8, 2, 0), ([129], 5, 1, 1 << 20)])
@pytest.mark.parametrize("c,x", [(60, -122), (-122, 60)])
def test_small_operands(lens, H, G, four, N, c, x, monkeypatch):
    """Operands near the smallest numbers against large ones: nothing of them is lost (the same bound)."""
    _compare(lens, H, G, four, N, 1.0, monkeypatch, 2.0 ** c, 2.0 ** x)


def _inputs(lens, H, G, N, speed=1.0, c_scale=1.0, x_scale=1.0):
    V = 64
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + H + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    T, off = sum(lens), 2 * G * N
    rec = rnd(T, -(-(off + H * V + 2 * H + G) // 4) * 4)
    rec[:, : G * N] *= c_scale
    rec[:, off: off + H * V] *= x_scale
    a_log, step = 0.3 * rnd(H), speed * torch.nn.functional.softplus(rnd(T, H))
    rec[:, off + H * V: off + H * V + H] = torch.exp(-torch.exp(a_log) * step)
    rec[:, off + H * V + H: off + H * V + 2 * H] = step
    rec[:, off + H * V + 2 * H: off + H * V + 2 * H + G] = (rec[:, : G * N] * rec[:, G * N: off]).view(T, G, N).sum(-1)
    return rec, a_log, step, 0.3 * x_scale * rnd(len(lens), H * N * V)


def _run(rec, a_log, state, lens, H, G, N):
    from nanospec_b200 import ops
    from nanospec_b200.parts import Workspace
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    ws = Workspace(DEV)
    ctx = SimpleNamespace(n_requests=len(lens), extras={}, q_lens=lens, max_q_len=max(lens), state_slot=i32(list(range(len(lens)))),
                          qo_indptr=i32([sum(lens[:i]) for i in range(len(lens) + 1)]), buffer=lambda name, cols, dtype, rows: ws.get(name, rows, cols, dtype))
    out = torch.empty(sum(lens), H * 64, device=DEV)
    ops.ssm_scan(rec, a_log, state.clone(), ctx, out, H, G, N, 64)
    return out.view(-1, H, 64)


def _walk(rec, a_log, step, state, lens, H, G, N):
    """(y, the sum of its terms' sizes) of every token in 64 bits, token by token."""
    T, V, off = sum(lens), 64, 2 * G * N
    C, B = (rec[:, k * G * N: (k + 1) * G * N].double().view(T, G, N).repeat_interleave(H // G, 1) for k in (0, 1))
    x, dt = rec[:, off: off + H * V].double().view(T, H, V), step.double()
    decay, at, ys, sizes = torch.exp(-torch.exp(a_log.double()) * dt), 0, [], []
    for r, n in enumerate(lens):
        R = state[r].double().view(H, N, V)
        size = R.abs()
        for t in range(at, at + n):
            add = (dt[t, :, None] * B[t])[:, :, None] * x[t][:, None, :]
            R, size = decay[t][:, None, None] * R + add, decay[t][:, None, None] * size + add.abs()
            ys.append(torch.einsum("hn,hnv->hv", C[t], R))
            sizes.append(torch.einsum("hn,hnv->hv", C[t].abs(), size))
        at += n
    return torch.stack(ys), torch.stack(sizes)


def _compare(lens, H, G, four, N, speed, monkeypatch, c_scale=1.0, x_scale=1.0):
    from nanospec_b200 import ops
    monkeypatch.setattr(ops, "SSM_FOUR_HEADS_FROM", four)
    rec, a_log, step, state = _inputs(lens, H, G, N, speed, c_scale, x_scale)
    out = _run(rec, a_log, state, lens, H, G, N)
    y, most = _walk(rec, a_log, step, state, lens, H, G, N)
    for t in range(sum(lens)):
        assert bool(((out[t].double() - y[t]).abs() <= most[t] * 120 * 2.0 ** -24).all()), t


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("H,G,four", [(8, 2, 0), (3, 1, 1 << 20)])
def test_what_is_not_finite(H, G, four, N, monkeypatch):
    """An infinity or a NaN of one token's x stays out of the tokens before it and the features beside it, an infinity stays one within its
    chunk, a state's too; numbers beyond the parts' range count as they are.  Rows made from the floats stay within the bound."""
    from nanospec_b200 import ops
    monkeypatch.setattr(ops, "SSM_FOUR_HEADS_FROM", four)
    lens, off, inf = [150], 2 * G * N, float("inf")
    rec, a_log, step, state = _inputs(lens, H, G, N)
    y, most = _walk(rec, a_log, step, state, lens, H, G, N)
    bound = most * 120 * 2.0 ** -24
    near = lambda out, sel: bool(((out.double() - y).abs() <= bound)[sel].all())  # noqa: E731
    dot = torch.einsum("tgn,sgn->gts", rec[:, : G * N].double().view(-1, G, N), rec[:, G * N: off].double().view(-1, G, N))
    for t0, h, v in ((70, H - 1, 5), (100, 0, 63), (127, 1, 16)):  # in the second chunk, whose tokens are 64 .. 127
        bad = rec.clone()
        bad[t0, off + h * 64 + v] = inf
        out = _run(bad, a_log, state, lens, H, G, N)
        assert near(out, (slice(0, t0),))
        others = [(k, e) for k in range(H) for e in (0, 15, 16, 47) if (k, e) != (h, v)]
        assert all(near(out, (slice(None), k, e)) for k, e in others)
        seen = out[t0:128, h, v]
        alive = torch.exp(-torch.exp(a_log[h].double()) * torch.cat([step.new_zeros(1), step[t0 + 1:128, h]]).double().cumsum(0)) > 1e-30
        assert torch.equal(seen[alive].double(), torch.sign(dot[h // (H // G), t0:128, t0])[alive] * inf)
        bad[t0, off: off + H * 64] = float("nan")
        out = _run(bad, a_log, state, lens, H, G, N)
        assert near(out, (slice(0, t0),)) and bool(out[t0:].isnan().all())
    bad = state.clone()
    bad.view(H, N, 64)[H - 1, 3, 20] = inf
    out = _run(rec, a_log, bad, lens, H, G, N)
    assert near(out, (slice(None), slice(0, H - 1))) and near(out, (slice(None), H - 1, 21))
    assert torch.equal(out[:5, H - 1, 20], torch.sign(rec[:5, (G - 1) * N + 3]) * inf)
    large = rec.clone()
    large[:, : G * N] *= 2.0 ** -100
    large[:, off: off + H * 64] *= 2.0 ** 110
    large_state = state * 2.0 ** 110
    out, (y, most) = _run(large, a_log, large_state, lens, H, G, N), _walk(large, a_log, step, large_state, lens, H, G, N)
    assert bool(((out.double() - y).abs() <= most * 120 * 2.0 ** -24).all())
