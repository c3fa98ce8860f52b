"""The rules that choose between two kernels of the same result, at measured points on both their sides (us on a B200 in the comments)."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch


def _step(held, brings):
    """What the rules look at of a step."""
    return SimpleNamespace(extras={}, q_lens=brings, kv_lens=[a + n for a, n in zip(held, brings)], n_tokens=sum(brings), max_q_len=max(brings),
                           device=torch.device("cpu"))


@pytest.mark.parametrize("held,brings,nq,dim,tiles", [
    ([0], [2], 32, 64, False),                       # 6.2 by row, 13.4 in tiles
    ([0], [16], 32, 128, False),                     # 12.1, 21.9
    ([0], [128], 4, 32, False),                      # 26.5, 32.7
    ([1500], [2], 4, 32, False),                     # 277, 294
    ([0], [128], 32, 64, True),                      # 111, 37
    ([0], [300], 4, 64, True),                       # 121, 72
    ([1500], [2], 32, 64, True),                     # 488, 312
    ([200] * 8, [60] * 8, 4, 32, True),              # 100, 63
    ([0], [97], 16, 64, True),                       # 51, 30: the chain and the pairs take alike, neither hides the other
    ([0] * 4, [40] * 4, 16, 64, True),               # 45, 22
    ([1500, 900], [2, 1], 8, 128, True),             # a request that brings one token does not count
])
def test_float32_portions(held, brings, nq, dim, tiles):
    from nanospec_b200 import ops
    assert ops.f32_tiles_pay(_step(held, brings), nq, dim) == tiles


@pytest.mark.parametrize("held,brings,nq,two,m16", [
    ([0] * 64, [2] * 64, 8, False, True),            # 11.2 on m16n8k16, 19.9 on tcgen05
    ([0] * 64, [2] * 64, 32, True, True),            # 37.3, 45.1
    ([100] * 32, [60] * 32, 8, False, True),         # 13.1, 14.8
    ([0] * 32, [120] * 32, 8, False, True),          # 12.0, 13.1
    ([100] * 32, [60] * 32, 32, True, False),        # 47.8, 40.6
    ([100] * 32, [120] * 32, 8, False, False),       # 19.8, 17.4
    ([1000] * 16, [2] * 16, 32, True, False),        # 75.6, 55.2
    ([0] * 16, [2] * 16, 8, False, False),           # 5.9, 5.8: a block an SM
    ([0] * 16, [180] * 16, 32, True, False),         # 43.0, 26.7
    ([1000] * 16, [1] * 16, 32, True, False),        # nothing but decoding
])
def test_prefill_of_many_short_portions(held, brings, nq, two, m16):
    from nanospec_b200 import ops
    ctx, blocks = _step(held, brings), sum(-(-n // 256) for n in brings if n > 1) * (nq // 2 if two else nq)
    assert ops.many_short_portions(ctx, blocks, 64, two, 148) == m16
    assert not ops.many_short_portions(ctx, blocks, 128, two, 148)


@pytest.mark.parametrize("held,brings,heads,rank,rot,window,unfolded", [
    # folded, unfolded
    ([500] + [300] * 8, [130] + [1] * 8, 16, 512, 64, 0, False),      # 65.6, 90.1
    ([8000, 500], [256, 1], 16, 256, 0, 1024, False),                 # 81.9, 109.0
    ([2000, 500], [512, 1], 16, 256, 0, 1024, False),                 # 122, 129
    ([2000, 500], [512, 1], 16, 512, 64, 1024, True),                 # 214, 135
    ([500] + [300] * 8, [130] + [1] * 8, 128, 512, 64, 0, True),      # 311, 199
    ([0, 500], [1500, 1], 16, 128, 64, 0, True),                      # 220, 123
    ([500], [130], 16, 512, 64, 0, True),                             # alone: 65, 46
    ([0], [127], 16, 512, 64, 0, False),
])
def test_latents_of_long_portions(held, brings, heads, rank, rot, window, unfolded):
    from nanospec_b200 import ops
    ctx = _step(held, brings)
    lane = SimpleNamespace(k=torch.empty(0, dtype=torch.bfloat16))
    rows, all_long = ops.latent_unfold_rows(ctx, lane, heads, 128, rot, 128, rank, window, torch.bfloat16, 0.1)
    assert (rows > 0) == unfolded and all_long == (unfolded and min(brings) >= 128)


@pytest.mark.gpu
@pytest.mark.parametrize("nq,nkv,brings,entry", [(8, 8, 24, "ns_attention_prefill_kept"), (16, 2, 24, "ns_attention_prefill_kept"),
                                                 (8, 8, 200, "ns_attention_prefill_tc")])
def test_prefill_of_many_requests(nq, nkv, brings, entry, monkeypatch):
    """Windowed prompts of 24 requests through `ops.attention` on both sides of the rule; the two kernels agree to the roundings of the weights
    (16 bits) and of the output (2^-9 of itself)."""
    from nanospec_b200 import ops
    from nanospec_b200.engine import ModelRunner, StepEntry
    from nanospec_b200.parts import CacheNeed
    from test_parts_gpu import _Shell
    d, B = 64, 24
    runner = ModelRunner(_Shell(torch.bfloat16, [(CacheNeed(nkv, d, 0, 0, None), None)], 1024), B * (brings // 16 + 1), 16, B)
    for r in range(B):
        runner.begin(r)
    ctx, _, _ = runner.build_context([StepEntry(r, [1] * brings) for r in range(B)])
    lane, g = ctx.lanes[0], torch.Generator(device="cuda").manual_seed(nq)
    for store in (lane.k, lane.v):
        store.copy_(torch.randn(store.shape, generator=g, device="cuda"))
    qkv = torch.randn(B * brings, nq * d, generator=g, device="cuda").to(torch.bfloat16)
    names, call, outs = [], ops.lib.call, []
    monkeypatch.setattr(ops.lib, "call", lambda name, *a: (names.append(name), call(name, *a)))
    for rule in (ops.many_short_portions, lambda *a: entry == "ns_attention_prefill_tc"):  # the rule, and the other kernel
        monkeypatch.setattr(ops, "many_short_portions", rule)
        outs.append(torch.zeros(B * brings, nq * d, device="cuda", dtype=torch.bfloat16))
        ops.attention(qkv, lane, ctx, outs[-1], nq, nkv, d, d ** -0.5, window=100, keep_first=3, wide_weights=True)
    ops.check_kernel_errors()
    assert names[0] == entry and names[0] != names[1]
    assert float((outs[0].double() - outs[1].double()).norm() / outs[1].double().norm()) < 2.0 ** -8


def test_tiles_of_the_experts_products():
    """By the rows that an expert holds, and pairs of SMs only where there are tiles for them."""
    from nanospec_b200 import ops
    assert [ops.moe_tile(32, 32 * per, 1024) for per in (1, 24, 25, 119, 120, 600)] == [32, 32, 128, 128, 256, 256]
    assert [ops.moe_tile(E, 300 * E, 1024) for E in (1, 8, 9, 10)] == [128, 128, 256, 256]
    assert ops.moe_tile(16, 300 * 16, 512) == 128 and ops.moe_tile(20, 300 * 20, 512) == 256
