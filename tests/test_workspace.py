"""How scratch buffers grow."""

from __future__ import annotations

import torch


def test_a_buffer_doubles_only_while_it_is_small(monkeypatch):
    from nanospec_b200.parts import context
    monkeypatch.setattr(context, "GROWTH_SPARE_MAX", 1 << 12)
    ws = context.Workspace(torch.device("cpu"))
    size = lambda: next(iter(ws._bufs.values())).shape[0]  # noqa: E731
    for rows, held in ((3, 16), (17, 32), (33, 64), (65, 128), (129, 193), (193, 193), (1000, 1000), (1001, 1065), (1065, 1065)):
        got = ws.get("x", rows, 16, torch.float32)  # 64 bytes a row: at most 64 rows beyond what is asked
        assert got.shape == (rows, 16) and size() == held, rows
        assert len(ws._bufs) == 1
