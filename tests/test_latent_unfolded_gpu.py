"""Latent attention of long portions of prompts on keys and values formed, beside requests that stay folded, against plain attention in 64 bits."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("rot_dim,rank,heads", [(64, 64, 3), (0, 80, 2), (64, 512, 4)])
@pytest.mark.parametrize("window", [0, 40, 100, 777])
@pytest.mark.parametrize("kind", ["sink", "head", "feature"])
@pytest.mark.parametrize("brings", [[130, 1, 300, 5], [128, 129], [2, 127]])
def test_unfolded_latent_attention(rot_dim, rank, heads, window, kind, brings, monkeypatch):
    """Everything else in the pages is NaN, the pages that a window has passed included.  Bound: queries, keys, values, outputs and the
    attention's result are rounded to bfloat16 once each (2^-9 of the value), as in the folded form."""
    from nanospec_b200 import ops
    from nanospec_b200.config import PartSpec
    from nanospec_b200.engine import ModelRunner, StepEntry
    from nanospec_b200.parts import build_part
    from test_parts_gpu import _Shell
    monkeypatch.setattr(ops, "LATENT_UNFOLD_MIXED", 0.0)  # also where so few heads and keys are not worth it beside short requests
    H, d, dv, R, W = heads, 128, 128, rank, 256
    pos = PartSpec("rotary", {"head_dim": rot_dim, "dims": rot_dim, "base": 10000.0, "layout": "interleaved", "scaling": None}) if rot_dim else None
    part = build_part("mixer", PartSpec("latent_attention", {
        "hidden": W, "heads": H, "dim": d, "rot_dim": rot_dim, "v_dim": dv, "rank": R, "scale": (d + rot_dim) ** -0.5, "window": window, "eps": 1e-6,
        "sink": kind == "sink", "gate": False if kind == "sink" else kind, "position": pos}), torch.bfloat16, DEV)
    g = torch.Generator(device=DEV).manual_seed(R + H + window)
    w = {}
    for name, spec in part.weight_specs().items():
        t = torch.randn(spec.shape, generator=g, device=DEV)
        w[name] = 1 + 0.1 * t if spec.init == "gain" else t if spec.rule == "float32" else (t * spec.shape[-1] ** -0.5).to(torch.bfloat16)
    part.bind(dict(w))
    w = {k: v.double() for k, v in w.items()}
    held = [0, 70, 333, 600][: len(brings)]
    runner = ModelRunner(_Shell(torch.bfloat16, [(part.cache_need(), None)], 2048), 200, 16, 8)
    for r in range(len(brings)):
        runner.begin(r)
    runner.build_context([StepEntry(r, [1] * n) for r, n in enumerate(held) if n])
    ctx, _, _ = runner.build_context([StepEntry(r, [1] * n) for r, n in enumerate(brings)])
    lane = ctx.lanes[0]
    lane.k.fill_(float("nan"))
    x = torch.randn(sum(brings), W, generator=g, device=DEV).to(torch.bfloat16)
    wants, at = [], 0
    for r, (a, n) in enumerate(zip(held, brings)):
        kept = torch.randn(a, R + rot_dim, generator=g, device=DEV).to(torch.bfloat16)
        p = torch.arange(a, device=DEV)
        seen = p[p > a - window] if window else p
        lane.k[lane.block_table[r].long()[seen // 16], 0, seen % 16] = kept[seen]
        h = x[at: at + n].double()
        at += n
        here = torch.arange(a, a + n, device=DEV).double()

        def rotate(t):
            if not rot_dim:
                return t
            ang = here[:, None] * 10000.0 ** (-torch.arange(0, rot_dim, 2, device=DEV).double() / rot_dim)
            cos, sin = (f(ang).reshape(n, *([1] * (t.dim() - 2)), -1) for f in (torch.cos, torch.sin))
            out = torch.empty_like(t)
            out[..., 0::2], out[..., 1::2] = t[..., 0::2] * cos - t[..., 1::2] * sin, t[..., 1::2] * cos + t[..., 0::2] * sin
            return out
        q = (h @ w["q"].T).view(n, H, d + rot_dim)
        q = torch.cat([q[..., :d], rotate(q[..., d:])], dim=-1)
        dkv = h @ w["dkv"].T
        c = dkv[:, :R] / torch.sqrt((dkv[:, :R] ** 2).mean(-1, keepdim=True) + 1e-6) * w["dkv.norm"]
        lat = torch.cat([kept.double(), torch.cat([c, rotate(dkv[:, R:])], dim=-1)])
        k = torch.cat([(lat[:, :R] @ w["uk"].T).view(-1, H, d), lat[:, None, R:].expand(-1, H, rot_dim)], dim=-1)
        v = (lat[:, :R] @ w["uv"].T).view(-1, H, dv)
        i, j = torch.arange(a, a + n, device=DEV)[:, None], torch.arange(a + n, device=DEV)[None, :]
        s = (torch.einsum("qhd,khd->hqk", q, k) * (d + rot_dim) ** -0.5).masked_fill(~((j <= i) & ((i - j < window) | (window == 0))), -math.inf)
        if kind == "sink":
            s = torch.cat([s, w["sink"][:, None, None].expand(H, n, 1)], dim=-1)
        o = torch.einsum("hqk,khd->qhd", torch.softmax(s, dim=-1)[..., : a + n], v)
        if kind != "sink":
            gates = torch.sigmoid(h @ w["g"].T)
            o = o * (gates[:, :, None] if kind == "head" else gates.view(n, H, dv))
        wants.append(o.reshape(n, H * dv) @ w["o"].T)
    want = torch.cat(wants)
    names, call = [], ops.lib.call
    monkeypatch.setattr(ops.lib, "call", lambda name, *a: (names.append(name), call(name, *a)))
    got = part.forward(x, ctx, lane).double()
    assert ("ns_attention_latent_flat" in names) == (max(brings) >= 128) and ("ns_attention_latent_tc" in names) == (min(brings) < 128)
    torch.cuda.synchronize()
    ops.check_kernel_errors()
    assert bool(got.isfinite().all())
    assert float((got - want).norm() / want.norm()) < 8 * 2.0 ** -9  # about five roundings of 2^-9 / sqrt(3) each, doubled
