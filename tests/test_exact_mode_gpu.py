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
