"""Ruler spacings that suit lists do not reach the forests: their walks read all
of a gap (a path of 2^25 vertices took 17 ms at spacing 48, 2.9 at its own).
The launches and level sizes show which spacing a call used."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LISTS = dict(ruler_spacing=48, ruler_spacing_deep=50)


@pytest.fixture(scope="module")
def kb():
    import kascade_b200

    return kascade_b200


def _path(n):
    order = torch.randperm(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    par = torch.empty_like(order)
    par[order[1:]] = order[:-1]
    par[order[0]] = order[0]
    return par


def _launches(kb, run, **t):
    ctx = kb.Context()
    out = run(ctx, kb.GpuTuning(profile=True, **t))
    times, levels = ctx.kernel_times(), ctx.levels()
    ctx.close()
    return out, {k: v[1] for k, v in times.items()}, levels


@pytest.mark.parametrize("n", [4097, 300_007])
def test_one_forest(kb, n):
    par = _path(n)
    run = lambda ctx, t: kb.root_forest(par, ctx=ctx, tuning=t)
    own, own_launches, own_levels = _launches(kb, run)
    out, launches, levels = _launches(kb, run, **LISTS)
    assert levels == own_levels and launches == own_launches
    assert torch.equal(out[0], own[0]) and torch.equal(out[1], own[1])
    assert _launches(kb, run, ruler_spacing=2)[2][1] == (n + 1) // 2  # smaller ones still apply


@pytest.mark.parametrize("n", [4097, 300_007])
def test_pointer_doubling(kb, n):
    par = _path(n)
    run = lambda ctx, t: kb.rank_list(par, ctx=ctx, tuning=t, algorithm=kb.Algorithm.PointerDoubling)
    own, own_launches, _ = _launches(kb, run)
    for t in (LISTS, dict(ruler_spacing=2, ruler_spacing_deep=3)):
        out, launches, _ = _launches(kb, run, **t)
        assert launches == own_launches
        assert torch.equal(out[0], own[0]) and torch.equal(out[1], own[1])


def test_forests_of_a_batch(kb):
    sizes = np.array([100_003, 7, 64_000], np.int64)
    inp, _ = kb.gen_batch(sizes, np.full(3, kb.SEG_FOREST), seed=5)
    segs = kb.make_segments(sizes, np.full(3, kb.SEG_FOREST))
    run = lambda ctx, t: kb.rank_batch(inp, segs, ctx=ctx, tuning=t)
    own, own_launches, _ = _launches(kb, run)
    out, launches, _ = _launches(kb, run, **LISTS)
    assert launches == own_launches
    assert torch.equal(out[0], own[0]) and torch.equal(out[1], own[1])
