"""Batches of lists and forests around the sizes at which their two element
spaces change path: nothing of one kind, empty instances, one element, tiles
and one-CTA bounds, every instance against the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_util import dev32, dev64, host_u64

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kb():
    import kascade_b200

    return kascade_b200


def _batch(kb, oracle_mod, sizes, kinds, rng, weighted):
    parts, roots, ranks = [], [], []
    w = rng.integers(0, 1 << 32, int(sum(sizes)), dtype=np.uint64).astype(np.uint32) if weighted else None
    at = 0
    for i, (n, k) in enumerate(zip(sizes, kinds)):
        if n == 0:
            continue
        if k == kb.SEG_LIST:
            succ = np.empty(n, np.uint64)
            order = rng.permutation(n)
            succ[order[:-1]] = order[1:]
            succ[order[-1]] = order[-1]
            root, rank = oracle_mod.rank_list(succ, w[at:at + n] if weighted else None)
        else:
            succ = oracle_mod.gen_forest(n, i + 1, 0, max(1, min(n // 50, 3)))
            root, rank = oracle_mod.root_forest(succ)
        parts.append(succ)
        roots.append(root)
        ranks.append(rank)
        at += n
    return np.concatenate(parts), w, np.concatenate(roots), np.concatenate(ranks)


L, F = 0, 1


@pytest.mark.parametrize("sizes,kinds", [
    ([1], [L]), ([1], [F]), ([4096, 1], [F, L]), ([0, 5, 0, 4097, 0], [L, F, F, F, L]),
    ([14336, 4096], [L, F]), ([14337, 4097], [L, F]), ([30_001], [F]), ([30_001], [L]),
    ([700, 65_537, 3, 12_288, 1, 1, 90_001], [F, L, F, F, L, F, L]),
    ([17] * 3000, [L, F, F] * 1000), ([1] * 9000, [L, F] * 4500),
    ([1_200_000, 400_003, 800_001], [L, F, F]),
])
@pytest.mark.parametrize("weighted", [False, True])
def test_spaces(kb, oracle_mod, sizes, kinds, weighted):
    rng = np.random.default_rng(len(sizes) * 7 + sizes[0])
    seg = [kb.SEG_FOREST if k == F else kb.SEG_LIST for k in kinds]
    succ, w, root_o, rank_o = _batch(kb, oracle_mod, sizes, seg, rng, weighted)
    segs = kb.make_segments(np.array(sizes, np.int64), np.array(seg, np.int64))
    wd = dev32(w) if weighted else None
    for tuning in ({}, dict(level0_mode=2, base_case_size=300), dict(ruler_spacing=3, ruler_spacing_deep=9)):
        root, rank = kb.rank_batch(dev64(succ), segs, wd, tuning=kb.GpuTuning(**tuning))
        np.testing.assert_array_equal(host_u64(root), root_o)
        np.testing.assert_array_equal(host_u64(rank), rank_o)


def test_plan_replays_both_spaces(kb, oracle_mod):
    rng = np.random.default_rng(3)
    sizes, kinds = [50_000, 60_000, 700, 20_000], [kb.SEG_LIST, kb.SEG_FOREST, kb.SEG_LIST, kb.SEG_FOREST]
    succ, w, root_o, rank_o = _batch(kb, oracle_mod, sizes, kinds, rng, True)
    x = dev64(succ)
    plan = kb.BatchPlan(x, kb.make_segments(np.array(sizes, np.int64), np.array(kinds, np.int64)), dev32(w))
    for _ in range(3):
        root, rank = plan.launch()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(host_u64(root), root_o)
        np.testing.assert_array_equal(host_u64(rank), rank_o)
        root.zero_()
        rank.zero_()
    x[0] = 1 << 40  # out of range: reported by the replay, and gone with the next
    with pytest.raises(kb.KascadeError) as e:
        plan.launch()
    assert e.value.name == "OUT_OF_RANGE"
    x.copy_(dev64(succ))
    root, rank = plan.launch()
    np.testing.assert_array_equal(host_u64(rank), rank_o)


def test_status_of_calls_on_two_streams(kb, oracle_mod):
    """An async call's status is published before a call on another stream
    starts: that call's error is its own, and neither leaks into the next."""
    import ctypes

    rng = np.random.default_rng(5)
    sizes, kinds = [400_000, 300_000], [kb.SEG_LIST, kb.SEG_FOREST]
    succ, _, root_o, rank_o = _batch(kb, oracle_mod, sizes, kinds, rng, False)
    x, segs = dev64(succ), kb.make_segments(np.array(sizes, np.int64), np.array(kinds, np.int64))
    bad = dev64(np.array([1, 7, 2], np.uint64))
    good = dev64(np.array([1, 1, 1], np.uint64))
    ctx = kb.Context()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(20):
        with torch.cuda.stream(a):
            root, rank = kb.rank_batch(x, segs, tuning=kb.GpuTuning(async_=True), ctx=ctx)
        with torch.cuda.stream(b):
            with pytest.raises(kb.KascadeError) as e:
                kb.rank_list(bad, ctx=ctx)
            assert e.value.name == "OUT_OF_RANGE"
            assert kb.rank_list(good, ctx=ctx)[1].tolist() == [1, 0, 1]
        with torch.cuda.stream(a):
            root, rank = kb.rank_batch(x, segs, tuning=kb.GpuTuning(async_=True), ctx=ctx)
            kb._lib.check(kb.lib.kascade_ctx_sync(ctx.handle, ctypes.c_void_p(a.cuda_stream)), "kascade_ctx_sync", ctx.handle)
        np.testing.assert_array_equal(host_u64(root), root_o)
        np.testing.assert_array_equal(host_u64(rank), rank_o)
    ctx.close()
