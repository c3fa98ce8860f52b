"""The kernels of the float32 mode at the edges of their tiles and of the rules that choose among them."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("K", [4, 60, 132, 133])  # less than a k tile, not whole tiles, not whole pieces of four
@pytest.mark.parametrize("M,N", [
    (1, 33), (4, 31), (5, 64), (8, 95), (9, 65), (16, 130), (17, 64), (32, 40), (32, 9500),  # rows of x side by side
    (33, 63), (32, 9473), (63, 65), (65, 127), (100, 320),                                    # small tiles
    (2050, 3600), (770, 8961),                                                                # wide tiles
])
def test_gemm_f32_kernels_give_the_same_bits(M, N, K):
    """Every result is one chain of fmaf over k in ascending order, whatever kernel the sizes choose: rows and columns taken alone (other
    kernels, other tiles) have the same bits.  The bound against 64 bits: K roundings of half an ulp each of a partial sum below sum |x w|."""
    from nanospec_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M * 7 + N + K)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    out = torch.full((M, N + 3), 7.0, device=DEV)
    ops.linear(x, w, out[:, :N])
    bound = (x.abs().double() @ w.abs().double().T) * (K * 2.0 ** -24)
    assert bool(((out[:, :N].double() - x.double() @ w.double().T).abs() <= bound).all())
    assert bool((out[:, N:] == 7.0).all())  # nothing beside the result is touched
    for rows in {1, 7, 20, 48}:
        if rows < M:
            part = torch.empty(rows, N, device=DEV)
            ops.linear(x[M - rows:], w, part)
            assert torch.equal(part, out[M - rows:, :N]), rows
    # operands whose rows do not start on 16 bytes take plain loads
    wide = torch.zeros(M, K + 1, device=DEV)
    wide[:, 1:] = x
    odd = torch.empty(M, N, device=DEV)
    ops.linear(wide[:, 1:], w, odd)
    assert torch.equal(odd, out[:, :N])


@pytest.mark.parametrize("nq,nkv,d,dv,page", [(4, 4, 32, 32, 8), (8, 2, 64, 64, 16), (24, 8, 128, 128, 16), (32, 1, 20, 20, 8), (5, 1, 36, 100, 16),
                                             (6, 2, 256, 8, 8), (2, 1, 4, 256, 16), (66, 2, 16, 16, 8)])  # (the last: 33 heads to a kv head, the exact kernel's)
@pytest.mark.parametrize("options", ["plain", "sink", "gate", "features"])
def test_attention_f32_portions_give_the_exact_kernels_bits(nq, nkv, d, dv, page, options, monkeypatch):
    """Portions of unlike lengths on unlike contexts beside decode tokens through `ops.attention`, against the one-warp kernel over the
    same rows, bit for bit (that kernel is tested against plain attention); pages that nobody wrote hold NaN."""
    from nanospec_b200 import ops
    from nanospec_b200.engine import StepEntry
    from nanospec_b200.parts import CacheNeed
    from test_parts_gpu import _Shell
    from nanospec_b200.engine import ModelRunner
    held, brings = [0, 37, 5, 130, 64], [33, 1, 129, 1, 31]
    need = CacheNeed(nkv, d, 0, 0, None if dv == d else dv)
    runner = ModelRunner(_Shell(torch.float32, [(need, None)]), 128, page, 8)
    for r in range(5):
        runner.begin(r)
    runner.build_context([StepEntry(r, [1] * n) for r, n in enumerate(held) if n])
    ctx, _, _ = runner.build_context([StepEntry(r, [1] * n) for r, n in enumerate(brings)])
    lane = ctx.lanes[0]
    g = torch.Generator(device=DEV).manual_seed(nq + d + dv)
    lane.k.fill_(float("nan")), lane.v.fill_(float("nan"))
    for r, (a, n) in enumerate(zip(held, brings)):
        at = torch.arange(a + n, device=DEV)
        for store in (lane.k, lane.v):
            store[lane.block_table[r].long()[at // page], :, at % page] = torch.randn(a + n, nkv, store.shape[-1], generator=g, device=DEV)
    N = sum(brings)
    qkv = torch.randn(N, nq * d + 8, generator=g, device=DEV)
    extra = {"sink": dict(sink=torch.randn(nq, generator=g, device=DEV)), "gate": dict(gate=torch.randn(N, nq, generator=g, device=DEV)),
             "features": dict(gate=torch.randn(N, nq * dv, generator=g, device=DEV), feature_gate=True, out_scale=0.5, softcap=2.0)}.get(options, {})
    monkeypatch.setattr(ops, "F32_TILES", True)  # also where so few rows do not take them
    got, want = torch.empty(N, nq * dv, device=DEV), torch.empty(N, nq * dv, device=DEV)
    ops.attention(qkv, lane, ctx, got, nq, nkv, d, 0.3, v_dim=dv, **extra)
    ops.attention_generic(qkv, lane.k, lane.v, lane.block_table, ctx.token_req, ctx.positions, want, nq, nkv, d, page, 0.3, v_dim=dv, **extra)
    assert bool(want.isfinite().all()) and torch.equal(got, want)
