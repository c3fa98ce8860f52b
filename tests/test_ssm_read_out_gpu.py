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


def _compare(lens, H, G, four, N, speed, monkeypatch, c_scale=1.0, x_scale=1.0):
    from nanospec_b200 import ops
    from nanospec_b200.parts import Workspace
    monkeypatch.setattr(ops, "SSM_FOUR_HEADS_FROM", four)
    V = 64
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + H + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    T, off, per = sum(lens), 2 * G * N, H // G
    rec = rnd(T, -(-(off + H * V + 2 * H + G) // 4) * 4)
    rec[:, : G * N] *= c_scale
    rec[:, off: off + H * V] *= x_scale
    a_log, step = 0.3 * rnd(H), speed * torch.nn.functional.softplus(rnd(T, H))
    rec[:, off + H * V: off + H * V + H] = torch.exp(-torch.exp(a_log) * step)
    rec[:, off + H * V + H: off + H * V + 2 * H] = step
    rec[:, off + H * V + 2 * H: off + H * V + 2 * H + G] = (rec[:, : G * N] * rec[:, G * N: off]).view(T, G, N).sum(-1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    ws, state = Workspace(DEV), 0.3 * x_scale * rnd(len(lens), H * N * V)
    ctx = SimpleNamespace(n_requests=len(lens), extras={}, q_lens=lens, max_q_len=max(lens), state_slot=i32(list(range(len(lens)))),
                          qo_indptr=i32([sum(lens[:i]) for i in range(len(lens) + 1)]), buffer=lambda name, cols, dtype, rows: ws.get(name, rows, cols, dtype))
    S, out = state.clone(), torch.empty(T, H * V, device=DEV)
    ops.ssm_scan(rec, a_log, S, ctx, out, H, G, N, V)
    C, B = (rec[:, k * G * N: (k + 1) * G * N].double().view(T, G, N).repeat_interleave(per, 1) for k in (0, 1))
    x, dt = rec[:, off: off + H * V].double().view(T, H, V), step.double()
    decay, at = torch.exp(-torch.exp(a_log.double()) * dt), 0
    for r, n in enumerate(lens):
        R = state[r].double().view(H, N, V)
        size = R.abs()
        for t in range(at, at + n):
            add = (dt[t, :, None] * B[t])[:, :, None] * x[t][:, None, :]
            R, size = decay[t][:, None, None] * R + add, decay[t][:, None, None] * size + add.abs()
            y, most = torch.einsum("hn,hnv->hv", C[t], R), torch.einsum("hn,hnv->hv", C[t].abs(), size)
            assert bool(((out[t].double().view(H, V) - y).abs() <= most * 120 * 2.0 ** -24).all()), (r, t - at)
        at += n
