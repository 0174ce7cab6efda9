"""One partition pass over the write-free log, or two: the rule's edge, and that
sizes at which one pass is far slower (2^25 elements: 2.8 ms against 1.8) take
two.  Both give the stamping path's results."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

ONE_PASS_MAX = 3000 << 13


@pytest.mark.parametrize("n,two", [(ONE_PASS_MAX, False), (ONE_PASS_MAX + 1, True), (1 << 25, True)])
@pytest.mark.parametrize("layout", [0, 1])
def test_passes_by_size(n, two, layout):
    import kascade_b200 as kb

    succ, w = kb.gen_list(n, n, layout), kb.gen_weights(n, n + 1, 16)
    ctx = kb.Context()
    root, rank = kb.rank_list(succ, w, ctx=ctx, tuning=kb.GpuTuning(profile=True))
    assert ("partition" in ctx.kernel_times()) == two
    ctx.close()
    root_s, rank_s = kb.rank_list(succ, w, tuning=kb.GpuTuning(level0_mode=1))
    assert torch.equal(root, root_s) and torch.equal(rank, rank_s)
