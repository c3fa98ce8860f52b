"""The tcgen05 prefill attention with windows, kept first keys, chunks, weights of 16 bits, sinks and gates, against attention in 64 bits."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("nq,nkv,d", [(8, 2, 64), (3, 1, 64), (4, 2, 128)])  # two heads to a block (with 64), one, heads of 128
@pytest.mark.parametrize("page", [8, 16, 64])
@pytest.mark.parametrize("mask", ["window 5", "window 64 keep 3", "window 130 keep 70", "window 300 keep 200", "window 1000 keep 8", "chunk 96", "all"])
@pytest.mark.parametrize("options", ["plain", "wide sink", "wide gate", "features"])
def test_prefill_general(nq, nkv, d, page, mask, options, monkeypatch):
    """Portions on contexts whose pages behind the window hold NaN, as does everything that nobody wrote.  Bounds: a weight's rounding moves the
    output by at most 2^-9 of the largest value (2^-16 with wide weights), the output's own rounding by 2^-9 of itself."""
    from nanospec_b200 import ops
    from nanospec_b200.engine import ModelRunner, StepEntry
    from nanospec_b200.parts import CacheNeed
    from test_parts_gpu import _Shell
    words = mask.split()
    window = int(words[1]) if words[0] == "window" else 0
    keep = int(words[3]) if len(words) > 2 else 0
    chunk = int(words[1]) if words[0] == "chunk" else 0
    held, brings = [0, 37, 511, 190], [65, 300, 257, 2]
    runner = ModelRunner(_Shell(torch.bfloat16, [(CacheNeed(nkv, d, 0, 0, None), None)], 1024), 1400 // page + 8, page, 8)
    for r in range(4):
        runner.begin(r)
    runner.build_context([StepEntry(r, [1] * n) for r, n in enumerate(held) if n])
    ctx, _, _ = runner.build_context([StepEntry(r, [1] * n) for r, n in enumerate(brings)])
    lane = ctx.lanes[0]
    g = torch.Generator(device=DEV).manual_seed(nq + d + page + window)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    rest = 0.0 if (mask, options) == ("all", "plain") else float("nan")  # (the plain instance loads whole pages, finite values)
    lane.k.fill_(rest), lane.v.fill_(rest)
    first = lambda p: max(p - window + 1 if window else 0, p // chunk * chunk if chunk else 0, 0)  # noqa: E731
    N = sum(brings)
    qkv, scale = rnd(N, nq * d + 8) * 2, d ** -0.5
    wide = options.startswith("wide")
    extra = dict(wide_weights=wide)
    if "sink" in options:
        extra["sink"] = torch.randn(nq, generator=g, device=DEV) * 3
    if "gate" in options:
        extra["gate"] = rnd(N, nq)
    if options == "features":
        extra |= dict(gate=rnd(N, nq * d), feature_gate=True, out_scale=0.5)
    want, at = [], 0
    for r, (a, n) in enumerate(zip(held, brings)):
        k, v = rnd(a + n, nkv, d), rnd(a + n, nkv, d)
        pos = torch.arange(a + n, device=DEV)
        seen = pos[(pos >= first(a)) | (pos < keep)]  # what the first token's successors may still see; the rest has been given back
        for store, x in ((lane.k, k), (lane.v, v)):
            store[lane.block_table[r].long()[seen // page], :, seen % page] = x[seen]
        q = qkv[at: at + n, : nq * d].view(n, nq, d).double()
        i, j = torch.arange(a, a + n, device=DEV)[:, None], pos[None, :]
        lo = torch.tensor([first(p) for p in range(a, a + n)], device=DEV)[:, None]
        ok = (j <= i) & ((j >= lo) | (j < keep))
        for h in range(nq):
            s = (q[:, h] @ k[:, h // (nq // nkv)].double().T * scale).masked_fill(~ok, -math.inf)
            if "sink" in extra:
                s = torch.cat([s, extra["sink"][h].double().expand(n, 1)], dim=1)
            o = torch.softmax(s, dim=1)[:, : a + n] @ v[:, h // (nq // nkv)].double() * extra.get("out_scale", 1.0)
            if "gate" in extra:
                z = extra["gate"][at: at + n].double()
                o = o * torch.sigmoid(z[:, h * d: (h + 1) * d] if options == "features" else z[:, h: h + 1])
            want.append((at, h, o, v.abs().amax().double()))
        at += n
    for heads in ("always", "never"):
        monkeypatch.setattr(ops, "PREFILL_TWO_HEADS", heads)
        out = torch.full((N, nq * d + 8), 9.0, dtype=torch.bfloat16, device=DEV)
        ops.attention(qkv, lane, ctx, out[:, : nq * d], nq, nkv, d, scale, window, keep, None, chunk=chunk, **extra)
        torch.cuda.synchronize()
        ops.check_kernel_errors()
        assert bool((out[:, nq * d:] == 9.0).all())
        for row, h, o, top in want:
            got = out[row: row + o.shape[0], h * d: (h + 1) * d].double()
            err = (got - o).abs() - o.abs() * 2.0 ** -8
            assert float(err.max()) <= float(top) * 2.0 ** (-14 if wide else -8), (row, h)
