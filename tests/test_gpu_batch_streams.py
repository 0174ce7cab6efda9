"""Mixed batches on streams of every priority, in turn, and on the stream of an
SM partition: the results of the default stream."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def work():
    import kascade_b200 as kb

    sizes = np.array([200_003, 5, 90_001, 1, 40_000], np.int64)
    kinds = np.array([kb.SEG_LIST, kb.SEG_FOREST, kb.SEG_FOREST, kb.SEG_LIST, kb.SEG_LIST])
    inp, w = kb.gen_batch(sizes, kinds, seed=11)
    segs = kb.make_segments(sizes, kinds)
    root, rank = kb.rank_batch(inp, segs, w)
    torch.cuda.synchronize()
    return kb, inp, segs, w, root, rank


def _same(work, stream, ctx):
    kb, inp, segs, w, root, rank = work
    r, k = torch.full_like(root, -1), torch.full_like(rank, -1)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        kb.rank_batch(inp, segs, w, root_out=r, rank_out=k, ctx=ctx)
    torch.cuda.synchronize()
    assert torch.equal(r, root) and torch.equal(k, rank)


def test_priorities(work):
    ctx = work[0].Context()
    for priority in (-1, 0, -2, -2, -5, 0):
        _same(work, torch.cuda.Stream(priority=priority), ctx)
    ctx.close()


def test_partition(work):
    from cuda.bindings import driver as d

    def ok(r):
        assert r[0] == d.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    dev = ok(d.cuDeviceGet(torch.cuda.current_device()))
    sms = ok(d.cuDeviceGetDevResource(dev, d.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(d.cuDevSmResourceSplitByCount(1, sms, 0, 64))
    green = ok(d.cuGreenCtxCreate(ok(d.cuDevResourceGenerateDesc(groups, 1)), dev,
                                  d.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    s = ok(d.cuGreenCtxStreamCreate(green, d.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    ctx = work[0].Context()
    try:
        assert int(ok(d.cuStreamGetGreenCtx(s))) != 0
        _same(work, torch.cuda.ExternalStream(int(s)), ctx)
        _same(work, torch.cuda.Stream(), ctx)
        _same(work, torch.cuda.ExternalStream(int(s)), ctx)
    finally:
        ctx.close()
        torch.cuda.synchronize()
        d.cuStreamDestroy(s)
        d.cuGreenCtxDestroy(green)
