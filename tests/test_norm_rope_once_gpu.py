"""The norm, rotation and store of bfloat16 rows in one reading (csrc/rope_kv.cu) against the general kernel, which a bias of zeros takes."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("interleaved", [True, False])
@pytest.mark.parametrize("gains", [(True, True), (True, False), (False, False)])
@pytest.mark.parametrize("nq,nkv,d,dv,pairs,write", [
    (1, 1, 16, 8, 8, True),        # the smallest pieces
    (32, 8, 64, 64, 32, True),
    (12, 4, 128, 64, 32, True),    # half of a head passes
    (40, 8, 64, 128, 16, True),
    (16, 16, 128, 128, 64, True),  # 512 threads when interleaved
    (3, 0, 64, 64, 24, False),     # rows of q alone
    (5, 2, 32, 256, 16, True),     # more pieces of values than of heads
])
def test_one_reading(nq, nkv, d, dv, pairs, write, gains, interleaved):
    """Norms summed in another order move a result by one rounding of the product before it (2^-23) and so by one step of bfloat16 (2^-8) at
    most; without gains nothing is summed and the bits are the same.  A padding row is left alone."""
    from nanospec_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(nq * 100 + d + pairs)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    page, n = 8, 9
    ctx = SimpleNamespace(positions=i32([0, 1, 2, 700, 701, 3, 4, 2047, 0]), token_req=i32([0, 0, 0, 1, 1, 2, 2, 3, -1]))
    table = torch.randperm(4 * 260, generator=torch.Generator().manual_seed(1))[: 4 * 257].to(torch.int32).view(4, 257).to(DEV)
    width = nq * d + nkv * (d + dv)
    rows = rnd(n, width + 8).to(torch.bfloat16)
    freq = 1e4 ** (-torch.arange(pairs, device=DEV, dtype=torch.float32) / pairs)
    q_gain, k_gain = (1 + 0.1 * rnd(nq * d) if gains[0] else None), (1 + 0.1 * rnd(nkv * d) if gains[1] and nkv else None)
    got = []
    for bias in (None, torch.zeros(width, device=DEV)):
        x = rows.clone()
        lane = SimpleNamespace(k=torch.full((4 * 260, max(1, nkv), page, d), 7.0, device=DEV).to(torch.bfloat16),
                               v=torch.full((4 * 260, max(1, nkv), page, dv), 7.0, device=DEV).to(torch.bfloat16), block_table=table, page_size=page)
        ops.qk_norm_rope_store(x[:, :width], ctx, lane, freq, 1.25, interleaved, nq, nkv, d, dv, q_gain, k_gain, 1e-6, write, bias)
        got.append((x, lane.k, lane.v))
    for a, b in zip(*got):
        if any(gains):
            assert bool(((a.float() - b.float()).abs() <= b.float().abs() * 2.0 ** -8 + 2.0 ** -20).all())
        else:
            assert torch.equal(a, b)
    assert torch.equal(got[0][0][:, width:], rows[:, width:]) and torch.equal(got[0][0][8], rows[8])
    if write:
        assert torch.equal(got[0][2], got[1][2]) and bool((got[0][2] != 7.0).any())


def test_frequencies_just_written():
    """Frequencies from this library's kernel directly before: the rotation sees them."""
    from nanospec_b200 import ops
    n, heads, d = 64, 8, 64
    ctx = SimpleNamespace(positions=torch.arange(n, dtype=torch.int32, device=DEV), token_req=torch.zeros(n, dtype=torch.int32, device=DEV))
    rows = torch.randn(n, heads * d, device=DEV).to(torch.bfloat16)
    lane = SimpleNamespace(k=None, v=None, block_table=None, page_size=1)
    tables = [(1e4 ** (-torch.arange(32, device=DEV) / (8.0 + i))).to(torch.bfloat16).view(1, 32) for i in range(8)]
    freq, got, want = torch.empty(1, 32, device=DEV), [], []
    for out, late in ((want, False), (got, True)):
        for t in tables:
            x = rows.clone()
            torch.cuda.synchronize()
            ops.cast_f32(t, freq)
            if not late:
                torch.cuda.synchronize()
            ops.qk_norm_rope_store(x, ctx, lane, freq[0], 1.0, False, heads, 0, d, d, None, None, 1e-6, False)
            out.append(x)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
