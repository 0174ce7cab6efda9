"""A large list on a device with little memory left: the stamping path's
results, and the write-free path again when there is memory."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

N = (1 << 26) + 3


@pytest.mark.parametrize("in_place", [True, False])
def test_with_memory_for_stamps_only(in_place):
    import kascade_b200 as kb

    succ, w32 = kb.gen_list(N, 0x10, 0), kb.gen_weights(N, 0x11, 16)
    w = w32.long()
    root, rank = (succ.clone(), w.clone()) if in_place else (torch.empty_like(succ), torch.empty_like(w))
    ctx, kept = kb.Context(), None

    def run():
        if in_place:
            root.copy_(succ), rank.copy_(w)
            tuning = kb.SparseRulingSetConfig(gpu=kb.GpuTuning(profile=True))
            kb.sparse_ruling_set(tuning, root, rank, ctx=ctx)
        else:
            kb.rank_list(succ, w32, root_out=root, rank_out=rank, ctx=ctx, tuning=kb.GpuTuning(profile=True))
        kernels = set(ctx.kernel_times())
        ctx.reset_kernel_times()
        return kernels

    try:
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        kept = torch.empty(torch.cuda.mem_get_info()[0] - 24 * N, dtype=torch.uint8, device="cuda")
        for _ in range(2):
            assert "propagate" in run()  # (level 0's and the deeper levels' stamping path)
            assert not {"resolve", "place"} & run()
        del kept
        kept = None
        torch.cuda.empty_cache()
        first = root.clone(), rank.clone()
        assert {"resolve", "place"} <= run()
        assert torch.equal(root, first[0]) and torch.equal(rank, first[1])
        end = succ == torch.arange(N, device="cuda")
        own = torch.where(end, 0, w)
        rank = torch.where(end, 0, rank)
        assert bool((rank == torch.where(end, 0, own + rank[succ])).all()) and bool((root == root[succ]).all())
    finally:
        del kept
        ctx.close()
        torch.cuda.empty_cache()
