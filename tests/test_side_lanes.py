"""What a fork or a join asks of its own thread's next launch, other threads leave alone."""

from __future__ import annotations

import threading

import pytest
import torch


def _in_thread(fn):
    out = []
    t = threading.Thread(target=lambda: out.append(fn()))
    t.start()
    t.join()
    return out[0]


def test_a_full_launch_is_asked_of_one_thread():
    from nanospec_b200.ops import lib
    native = lib.load()

    def ask():
        native.ns_full_launch_next()
        return native.ns_full_launch_pending(), _in_thread(native.ns_full_launch_pending)
    assert _in_thread(ask) == (1, 0)
    assert native.ns_full_launch_pending() == 0


@pytest.mark.gpu
def test_another_threads_launch_does_not_take_it():
    from nanospec_b200 import ops
    from nanospec_b200.ops import lib
    native = lib.load()
    table, ids, out = torch.randn(8, 64, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda"), torch.empty(2, 64, device="cuda")

    def launch():
        ops.embed(table, ids, out)
        return native.ns_full_launch_pending()

    def ask():
        native.ns_full_launch_next()
        return _in_thread(launch), native.ns_full_launch_pending(), launch()
    assert _in_thread(ask) == (0, 1, 0)
