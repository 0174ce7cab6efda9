"""Lists of more than 2^31 elements, whose successors need all 32 bits of their
word: the write-free path's 16 B records, and the stamping path's with the stamp
inside.  Checked by the lists' own equations, a slice at a time."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

N = (1 << 31) + 4099


@pytest.mark.parametrize("mode", [0, 1])
def test_list(mode):
    import kascade_b200 as kb

    if torch.cuda.mem_get_info()[1] < 170 << 30:
        pytest.skip("needs a 180 GB device")
    torch.cuda.empty_cache()
    succ = kb.gen_list(N, 0x31, 0)
    ctx = kb.Context()
    root, rank = torch.empty_like(succ), torch.empty_like(succ)
    try:
        kb.rank_list(succ, root_out=root, rank_out=rank, ctx=ctx, tuning=kb.GpuTuning(level0_mode=mode))
    finally:
        ctx.close()
    step, ends, total = 1 << 27, 0, 0
    for a in range(0, N, step):
        s = succ[a:a + step]
        end = s == torch.arange(a, a + s.numel(), device="cuda")
        ends += int(end.sum())
        total += int(rank[a:a + step].sum())
        assert bool((rank[a:a + step] == torch.where(end, 0, 1 + rank[s])).all())
        assert bool((root[a:a + step] == root[s]).all())
        assert bool((root[a:a + step][end] == s[end]).all())
    assert ends == 1 and total == N * (N - 1) // 2  # one list: ranks 0 .. N - 1
