"""The experts' products in tiles of 256 rows on pairs of SMs (csrc/moe_tcgen05.cu) where a pair takes many tiles."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def _products(counts, width, ff, tiles, seed):
    """ys of both products for every tile size, and the rows in use."""
    from nanospec_b200 import ops
    E, n = len(counts), sum(counts)
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    xs, w_gate_up, w_down = rnd(n + 5, width), rnd(E, 2 * ff, width) * width ** -0.5, rnd(E, width, ff) * ff ** -0.5
    xs[n:] = float("nan")
    offsets = torch.tensor([sum(counts[:e]) for e in range(E + 1)], dtype=torch.int32, device=DEV)
    out = []
    for tile in tiles:
        act, ys = torch.full((n + 5, ff), float("nan"), dtype=torch.bfloat16, device=DEV), torch.full((n + 5, width), float("nan"), dtype=torch.bfloat16, device=DEV)
        old, ops.MOE_TILE = ops.MOE_TILE, tile
        try:
            for _ in range(3):
                ops.moe_grouped_tc(xs, offsets, w_gate_up, w_down, act, ys)
        finally:
            ops.MOE_TILE = old
        assert bool(ys[n:].isnan().all()) and bool(act[n:].isnan().all())
        out.append((act[:n], ys[:n]))
    ops.check_kernel_errors()
    return xs, w_gate_up, w_down, offsets, out


@pytest.mark.parametrize("counts", [
    [0, 1, 31, 32, 33, 255, 256, 257, 600, 900, 1200, 1500, 1800, 2000, 1000, 0],  # five tiles and more to a pair in the first product
    [9000],                                                                        # one expert: every pair at its rows
    [33] * 200,                                                                    # the second accumulator's and the first one's tiles of one chunk and a row
])
@pytest.mark.parametrize("width,ff", [(1032, 1024), (72, 640)])  # ragged last tiles of weights and of k; products shorter than the ring
def test_many_tiles_to_a_pair(counts, width, ff):
    """The bits of the tiles of 128 rows (the products' order over k is the same), and the products themselves against 64 bits: rounded to bfloat16, from
    sums of 2^-23 a term."""
    xs, w_gate_up, w_down, offsets, ((act, ys), (act2, ys2)) = _products(counts, width, ff, (256, 128), len(counts) + width)
    assert torch.equal(act, act2) and torch.equal(ys, ys2)
    for e, n in enumerate(counts):
        if n:
            at = int(offsets[e])
            want = act[at:at + n].double() @ w_down[e].double().T
            size = act[at:at + n].abs().double() @ w_down[e].abs().double().T
            assert bool(((ys[at:at + n].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * ff * 2.0 ** -23).all()), e


def test_more_experts_than_a_pair_counts():
    """Above 1,024 experts tiles of 256 become tiles of 128: the bits of tiles of 32."""
    counts = [(7 * e) % 5 for e in range(1030)]
    *_, ((act, ys), (act2, ys2)) = _products(counts, 64, 64, (256, 32), 3)
    assert torch.equal(act, act2) and torch.equal(ys, ys2)
