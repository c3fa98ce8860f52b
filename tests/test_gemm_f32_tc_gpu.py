"""The float32 product on the tensor cores (csrc/gemm_f32_tc.cu) at the edges of its tiles, splits and groups."""

from __future__ import annotations

import random

import pytest
import torch

DEV = "cuda"


def test_f32_tiles_fit():
    """What the kernel's entry demands of a split, over sizes spread by their logarithm."""
    from nanospec_b200 import ops
    rng = random.Random(5)
    for _ in range(2000):
        M, N, K = (int(2 ** rng.uniform(0, hi)) for hi in (14, 17, 14))
        rows, splits = ops.f32_tiles(M, N, K, 148)
        blocks = -(-K // 64)
        groups = -(-blocks // -(-blocks // min(8, -(-blocks // 8))))
        assert rows % 16 == 0 and 16 <= rows <= 96 and rows < M + 16
        assert splits == 1 or (splits <= groups and -(-N // 128) * -(-M // rows) * splits <= 148 and -(-groups // splits) * rows <= 96)


def test_f32_runs():
    """The runs cover the rows once, in whole tiles but for the last, and their parts stay below the limit; a product of few rows is one run."""
    from nanospec_b200 import ops
    for M, K in ((1, 1024), (641, 8192), (16384, 14336), (100000, 1028), (500, 1 << 20), (200, 1 << 24)):
        runs = ops.f32_runs(M, K, ops.F32_PARTS_MAX)
        assert [m for m, _ in runs] == [0, *(m + n for m, n in runs[:-1])] and sum(n for _, n in runs) == M
        assert all(n % 96 == 0 for _, n in runs[:-1])
        assert runs[0][1] <= 96 or 6 * runs[0][1] * K <= ops.F32_PARTS_MAX
        assert len(runs) == 1 or 6 * M * K > ops.F32_PARTS_MAX // 2
    assert ops.f32_runs(0, 1024, 1) == []


def _operands(M, N, K, seed, spread=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    if spread:
        x = x * torch.exp2(torch.randint(-spread, spread, (M, K), generator=g, device=DEV).float())
    return x, w


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1024, 1028, 1092, 4160])  # whole groups; four past a block; a ragged last block; groups of unlike lengths
@pytest.mark.parametrize("M,N", [(1, 1), (15, 127), (16, 128), (17, 129), (33, 300), (97, 260), (130, 20000)])
def test_f32_tc_product(M, N, K):
    """Against 64 bits: an element's products lose 2^-24 of themselves; a block's 24 additions truncate (2^-23 of what they reach), the K / 64 sums of
    blocks and groups round.  And no further off, in the 2-norm, than the chain of fmaf.  Every tile and split, rows alone and rows that
    do not start on 16 bytes give the same bits; nothing beside the result is touched."""
    from nanospec_b200 import ops
    from nanospec_b200.ops import lib
    x, w = _operands(M, N, K, M + N + K, spread=20 if M == 33 else 0)
    out = torch.full((M, N + 3), 7.0, device=DEV)
    ops.linear(x, w, out[:, :N])
    ref, size = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    err = out[:, :N].double() - ref
    assert bool((err.abs() <= size * (50 + K // 64 + 8) * 2.0 ** -24).all())
    assert bool((out[:, N:] == 7.0).all())
    if M * N > 1000:  # (a 2-norm of few elements is chance: here the chain's is five times as large or more)
        chain = torch.empty(M, N, device=DEV)
        lib.call("ns_gemm_f32", x.data_ptr(), w.data_ptr(), chain.data_ptr(), M, N, K, K, K, N, ops.sm_count(), ops._stream())
        assert float(err.norm()) <= float((chain.double() - ref).norm())
    got = torch.empty(M, N, device=DEV)
    blocks = -(-K // 64)
    groups = -(-blocks // -(-blocks // min(8, -(-blocks // 8))))
    for rows in (16, 32, 48, 96):
        for splits in (1, 2, 4):
            if splits == 1 or (splits <= groups and -(-N // 128) * -(-M // rows) * splits <= ops.sm_count() and -(-groups // splits) * rows <= 96):
                ops.linear_f32_tc(x, w, got.fill_(float("nan")), (rows, splits))
                assert torch.equal(got, out[:, :N]), (rows, splits)
    one = torch.empty(1, N, device=DEV)
    for m in {0, M // 2, M - 1}:
        ops.linear(x[m:m + 1], w, one)
        assert torch.equal(one[0], out[m, :N])
    wide = torch.zeros(M, K + 1, device=DEV)
    wide[:, 1:] = x
    ops.linear(wide[:, 1:], w, got)
    assert torch.equal(got, out[:, :N])
    ops.check_kernel_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("tiles", [(16, 1), (16, 2), (48, 1)])
def test_f32_tc_infinities_and_ends_of_the_range(tiles):
    """An element whose floats have no parts (an infinity, a NaN, the largest numbers) is what the floats themselves give, subnormal results are
    as near as their spacing lets them be; every other element keeps its bits."""
    from nanospec_b200 import ops
    x, w = _operands(40, 200, 1024, 3)
    clean = torch.empty(40, 200, device=DEV)
    ops.linear_f32_tc(x, w, clean, tiles)
    y = x.clone()
    y[3, 7], y[5, 100], y[9] = float("nan"), float("inf"), 0.0
    y[12] *= 2.0 ** -124  # results of these are subnormal or nearly
    y[14, 0] = 3.4e38     # rounds to an infinite bfloat16
    v = w.clone()
    v[:, 0] *= 2.0 ** -10
    v[17, 5] = float("-inf")
    got = torch.empty(40, 200, device=DEV)
    ops.linear_f32_tc(y, v, got, tiles)
    assert bool(got[3].isnan().all())
    assert torch.equal(got[5, :17], torch.sign(v[:17, 100]) * float("inf"))
    assert bool((got[9, :17] == 0).all()) and bool(got[9, 17].isnan())  # 0 * -inf
    assert torch.equal(got[[0, 20, 39], 17], torch.sign(y[[0, 20, 39], 5]) * float("-inf"))
    keep = [c for c in range(200) if c != 17]
    for m in (12, 14):
        ref, size = y[m].double() @ v.double().T, y[m].abs().double() @ v.abs().double().T
        # a chain of 32 fmaf and five sums, or the bound above; numbers below 2^-126 are whole multiples of 2^-149
        assert bool(((got[m].double() - ref).abs()[keep] <= size[keep] * 82 * 2.0 ** -24 + 2.0 ** -143).all())
    same = torch.empty(40, 200, device=DEV)
    ops.linear_f32_tc(x, v, same, tiles)
    rows = [m for m in range(40) if m not in (3, 5, 9, 12, 14)]
    assert torch.equal(got[rows][:, keep], same[rows][:, keep])
    ops.check_kernel_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("tiles", [(16, 1), (16, 2), (48, 1)])
@pytest.mark.parametrize("small,large", [(-109, 40), (-112, 60), (-124, 60), (-136, 80), (-146, 100), (50, 50), (-100, -20)])
def test_f32_tc_small_and_large_operands(small, large, tiles):
    """Small numbers on either side lose nothing, whatever the results are, zeros among them stay zeros, and sums beyond the parts' range come
    from the floats: the bounds above (a chain of 32 fmaf and its five sums is below them)."""
    from nanospec_b200 import ops
    x, w = _operands(40, 200, 1024, 4)
    x[7], w[11] = 0.0, 0.0
    got = torch.empty(40, 200, device=DEV)
    for a, b in ((small, large), (large, small)):
        u, v = torch.ldexp(x, torch.tensor(a, device=DEV)), torch.ldexp(w, torch.tensor(b, device=DEV))
        ops.linear_f32_tc(u, v, got, tiles)
        ref, size = u.double() @ v.double().T, u.abs().double() @ v.abs().double().T
        assert bool(((got.double() - ref).abs() <= size * 82 * 2.0 ** -24 + 2.0 ** -149).all())
    ops.check_kernel_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("terms", [1, 2, 8])
def test_f32_tc_rows_of_few_terms(terms):
    """Rows of x that are zero but for a few numbers: a product leaves out 2^-24 of itself, each of its high by high steps truncates once (2^-23 of
    what is reached) and its block's sum joins with a rounding; what the small products truncate is a sixteenth of that."""
    from nanospec_b200 import ops
    x, w = _operands(70, 300, 2048, terms)
    order = torch.rand(70, 2048, generator=torch.Generator().manual_seed(terms)).argsort(1).to(DEV)
    x = torch.where(order < terms, x, 0.0)
    got = torch.empty(70, 300, device=DEV)
    ops.linear(x, w, got)
    ref, size = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    assert bool(((got.double() - ref).abs() <= size * (1 + 3.2 * terms) * 2.0 ** -24).all())
    ops.check_kernel_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,tiles", [(1, 128, 1024, (16, 2)), (33, 300, 1092, (48, 1)), (97, 257, 2048, (96, 1)), (20, 20000, 1024, (32, 1))])
def test_f32_tc_weights_of_16_bits(M, N, K, tiles):
    """Products with parts of w that are zero are left out: such weights' elements stay within the bound, and keep their bits when another row of w's tile,
    in its first or last block of k, has all three parts (then none are left out)."""
    from nanospec_b200 import ops
    x, w = _operands(M, N, K, M + N)
    w = w.bfloat16().float()
    got, other = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.linear_f32_tc(x, w, got, tiles)
    ref, size = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    assert bool(((got.double() - ref).abs() <= size * (50 + K // 64 + 8) * 2.0 ** -24).all())
    for n, k in ((0, 0), (N // 2, K - 1), (N - 1, 64)):
        v = w.clone()
        v[n, k] += 2.0 ** -18
        assert float(v[n, k]) != float(w[n, k])
        ops.linear_f32_tc(x, v, other, tiles)
        keep = [c for c in range(N) if c != n]
        assert torch.equal(got[:, keep], other[:, keep])
        ref = x.double() @ v[n].double()
        assert bool(((other[:, n].double() - ref).abs() <= size[:, n] * 1.01 * (50 + K // 64 + 8) * 2.0 ** -24).all())
    ops.check_kernel_errors()


@pytest.mark.gpu
def test_f32_tc_late_weights():
    """Weights from DRAM, whose tiles land out of order: the bits of the first run again and again (odd and even rings of w's tiles)."""
    from nanospec_b200 import ops
    x, w = _operands(3, 32768, 2048, 1)
    flush = torch.empty(64 << 20, device=DEV)
    first, got = torch.empty(3, 32768, device=DEV), torch.empty(3, 32768, device=DEV)
    for tiles in ((16, 1), (48, 1)):
        ops.linear_f32_tc(x, w, first, tiles)
        for _ in range(12):
            flush.zero_()
            ops.linear_f32_tc(x, w, got, tiles)
            assert torch.equal(got, first)
    ops.check_kernel_errors()


@pytest.mark.gpu
def test_f32_tc_weights_just_written():
    """w from this library's kernel directly before the product, one that starts its successor at once: the product sees all of it."""
    from nanospec_b200 import ops
    rounds = [_operands(8, 4096, 2048, seed) for seed in range(6)]
    rounds = [(x, w.bfloat16()) for x, w in rounds]
    want = []
    for x, w in rounds:
        want.append(torch.empty(8, 4096, device=DEV))
        w32 = w.float()
        torch.cuda.synchronize()
        ops.linear(x, w32, want[-1])
    w32, got = torch.empty(4096, 2048, device=DEV), [torch.empty(8, 4096, device=DEV) for _ in rounds]
    torch.cuda.synchronize()
    for (x, w), out in zip(rounds, got):
        ops.cast_f32(w, w32)
        ops.linear(x, w32, out)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    ops.check_kernel_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("M", [97, 192, 300])
def test_f32_tc_rows_in_runs(M, monkeypatch):
    """More rows than the parts' limit go in runs, with the same bits, rows of x apart and on odd addresses too."""
    from nanospec_b200 import ops
    x, w = _operands(M, 260, 1028, M)
    want, got = torch.empty(M, 260, device=DEV), torch.full((M, 263), 7.0, device=DEV)
    ops.linear(x, w, want)
    monkeypatch.setattr(ops, "F32_PARTS_MAX", 1 << 20)
    assert len(ops.f32_runs(M, 1028, ops.F32_PARTS_MAX)) > 1
    wide = torch.zeros(M, 1033, device=DEV)
    wide[:, 3:1031] = x
    for rows in (x, wide[:, 3:1031]):
        ops.linear(rows, w, got[:, :260].fill_(float("nan")))
        assert torch.equal(got[:, :260], want) and bool((got[:, 260:] == 7.0).all())
    ops.check_kernel_errors()
