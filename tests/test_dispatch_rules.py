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
    ([1500, 900], [2, 1], 8, 128, True),             # a request that brings one token does not count
])
def test_float32_portions(held, brings, nq, dim, tiles):
    from nanospec_b200 import ops
    assert ops.f32_tiles_pay(_step(held, brings), nq, dim) == tiles
