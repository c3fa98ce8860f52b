"""The delta rule's preparation with four channels to a thread against the one that takes a channel alone, bit for bit."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lens,G,H,D,V", [([1, 2, 3, 4, 5], 2, 4, 128, 128), ([300], 1, 1, 2, 4), ([1], 16, 32, 128, 128), ([7, 40], 3, 6, 20, 34)])
def test_wide_rows_give_the_same_bits(lens, G, H, D, V, dtype):
    from nanospec_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + H + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    T, C, s_floats, Dp = sum(lens), 2 * G * D + H * V, 64, ops.scan_padded_dim(D)
    width = -(-(C + 2 * H) // 8) * 8
    proj, taps = rnd(T, width).to(dtype), rnd(C, 4)
    a_log, dt_bias = 0.5 * rnd(H), rnd(H)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    ctx = SimpleNamespace(n_requests=len(lens), token_req=i32([r for r, n in enumerate(lens) for _ in range(n)]),
                          state_slot=i32([len(lens) - i for i in range(len(lens))]), qo_indptr=i32([sum(lens[:i]) for i in range(len(lens) + 1)]))
    state = rnd(len(lens) + 1, s_floats + 3 * C)
    cols = -(-(2 * G * Dp + H * V + 2 * H + G) // 4) * 4

    def run(p):
        S, rec = state.clone(), torch.full((T, cols), 7.0, device=DEV)
        ops.delta_prepare(p, taps, a_log, dt_bias, S, s_floats, ctx, rec, G, H, D, V, C, C + H, D ** -0.5, 1e-6)
        return rec, S

    odd = torch.empty(T, width + 1, dtype=dtype, device=DEV)  # rows that start anywhere: a channel to a thread
    odd[:, 1:] = proj
    rec, S = run(proj)
    rec1, S1 = run(odd[:, 1:])
    assert torch.equal(rec, rec1) and torch.equal(S, S1)
    assert bool((rec[:, 2 * G * Dp + H * V + 2 * H + G:] == 7.0).all())
