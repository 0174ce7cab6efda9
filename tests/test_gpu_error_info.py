"""A list ranker given branches names the first element with two predecessors,
by its place in the caller's arrays, on every path."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_util import dev64

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kb():
    import kascade_b200

    return kascade_b200


def _branched(n, branches, seed):
    """One list of half the elements; the rest in equal branches, each ending at
    an element of it.  Also the first of those elements."""
    rng = np.random.default_rng(seed)
    order = rng.permutation(n)
    main, rest = order[:n // 2], np.array_split(order[n // 2:], branches)
    succ = np.empty(n, np.int64)
    succ[main[:-1]], succ[main[-1]] = main[1:], main[-1]
    ends = main[rng.integers(1, len(main) - 1, branches)]
    for b, end in zip(rest, ends):
        succ[b[:-1]], succ[b[-1]] = b[1:], end
    return succ, int(ends.min())


def _info(kb, ctx, run):
    with pytest.raises(kb.KascadeError) as e:
        run()
    assert e.value.name == "NOT_A_LIST"
    return kb._lib.lib.kascade_ctx_error_info(ctx.handle)


@pytest.mark.parametrize("n", [8193, 14_336, 14_337, 100_003, 3_000_000, 6_000_001, 9_000_001])
def test_rank_list(kb, n):
    succ, first = _branched(n, 200, n)
    s, ctx = dev64(succ.astype(np.uint64)), kb.Context()
    w = torch.ones(n, dtype=torch.int32, device="cuda")
    for mode in (0, 1, 2):
        for weights in (None, w):
            t = kb.GpuTuning(level0_mode=mode)
            assert _info(kb, ctx, lambda: kb.rank_list(s, weights, ctx=ctx, tuning=t)) == first
    copy, rank = s.clone(), torch.ones_like(s)
    assert _info(kb, ctx, lambda: kb.sparse_ruling_set(kb.SparseRulingSetConfig(), copy, rank, ctx=ctx)) == first
    good = kb.gen_list(n, 1, 0)  # the next call is not the worse for it
    kb.rank_list(good, ctx=ctx)
    assert kb._lib.lib.kascade_ctx_error_info(ctx.handle) == 0
    ctx.close()


@pytest.mark.parametrize("sizes", [[9000], [300_000]])
def test_batch_and_plan(kb, sizes):
    n = sizes[0]
    succ, first = _branched(n, 100, n)
    before = kb.gen_forest(777, 1, 0, 3, 0)
    lists = kb.gen_list(1234, 2, 0)
    inp = torch.cat([before, lists, dev64(succ.astype(np.uint64)), before])
    segs = kb.make_segments(np.array([777, 1234, n, 777], np.int64),
                            np.array([kb.SEG_FOREST, kb.SEG_LIST, kb.SEG_LIST, kb.SEG_FOREST]))
    ctx = kb.Context()
    for mode in (0, 2):
        run = lambda: kb.rank_batch(inp, segs, ctx=ctx, tuning=kb.GpuTuning(level0_mode=mode))
        assert _info(kb, ctx, run) == first + 777 + 1234
    ctx.close()
    good = inp.clone()
    good[777 + 1234:777 + 1234 + n] = kb.gen_list(n, 3, 0)
    root, rank = (t.clone() for t in kb.rank_batch(good, segs))
    held = good.clone()
    plan = kb.BatchPlan(held, segs)
    for contents, ok in ((good, True), (inp, False), (inp, False), (good, True)):
        held.copy_(contents)
        if ok:
            r, k = plan.launch()
            assert torch.equal(r, root) and torch.equal(k, rank)
        else:
            with pytest.raises(kb.KascadeError) as e:
                plan.launch()
            assert e.value.name == "NOT_A_LIST"
    plan.close()


def test_async(kb):
    n = 50_000
    succ, first = _branched(n, 100, n)
    s, ctx = dev64(succ.astype(np.uint64)), kb.Context()
    kb.rank_list(s, ctx=ctx, tuning=kb.GpuTuning(async_=True))
    assert _info(kb, ctx, ctx.sync) == first
    kb.rank_list(s, ctx=ctx, tuning=kb.GpuTuning(async_=True))
    ctx.reserve(1 << 30)  # takes the records away before the error is read
    with pytest.raises(kb.KascadeError) as e:
        ctx.sync()
    assert e.value.name == "NOT_A_LIST"
    ctx.close()
