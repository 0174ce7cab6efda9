"""Level 0's record formats and paths at the sizes where the rule changes them:
records with stamps beside them, stamps inside, write-free with one and with
two partition passes; unit, 32-bit and 64-bit weights, in place and not.  The
paths agree with each other and with the lists' own equations."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_util import dev64, host_i64

pytestmark = pytest.mark.gpu

L2_BYTES = 88 << 20  # records and stamps beside each other up to here


@pytest.fixture(scope="module")
def kb():
    import kascade_b200

    return kascade_b200


def _lists(n, parts, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    order = torch.randperm(n, device="cuda", generator=g)
    ends = torch.zeros(n, dtype=torch.bool, device="cuda")
    ends[torch.randint(n, (parts - 1,), device="cuda", generator=g)] = True
    ends[-1] = True
    succ = torch.empty_like(order)
    succ[order] = torch.where(ends, order, torch.roll(order, -1))
    return succ


def _holds(succ, w, root, rank):
    """rank = own weight + the successor's rank, root = the successor's; ends: themselves, 0."""
    idx = torch.arange(succ.numel(), device="cuda")
    end = succ == idx
    assert bool((root[end] == idx[end]).all()) and bool((rank[end] == 0).all())
    own = torch.ones_like(rank) if w is None else w
    assert bool((rank == torch.where(end, 0, own + rank[succ])).all())
    assert bool((root == root[succ]).all())


@pytest.mark.parametrize("n", [L2_BYTES // 24, L2_BYTES // 24 + 1, L2_BYTES // 16, L2_BYTES // 16 + 1, 7_999_999,
                               8_000_000, (1 << 25) - 5, (1 << 25) + 1])
@pytest.mark.parametrize("wbits", [0, 32])
def test_sizes_of_the_rule(kb, n, wbits):
    succ = _lists(n, 5, n)
    w32 = kb.gen_weights(n, n + 1, wbits) if wbits else None
    w = None if w32 is None else w32.long() & 0xFFFFFFFF
    root, rank = kb.rank_list(succ, w32)
    _holds(succ, w, root, rank)
    for mode in (1, 2):
        r, k = kb.rank_list(succ, w32, tuning=kb.GpuTuning(level0_mode=mode))
        assert torch.equal(r, root) and torch.equal(k, rank), mode


@pytest.mark.parametrize("n", [L2_BYTES // 32, L2_BYTES // 32 + 1, 11_999_999, 12_000_000])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_in_place_64_bit_weights(kb, n, mode):
    succ = _lists(n, 7, n)
    g = torch.Generator(device="cuda")
    g.manual_seed(n + 3)
    w = torch.randint(-(1 << 60), 1 << 60, (n,), device="cuda", generator=g)
    root, rank = succ.clone(), w.clone()
    kb.sparse_ruling_set(kb.SparseRulingSetConfig(gpu=kb.GpuTuning(level0_mode=mode)), root, rank)
    end = succ == torch.arange(n, device="cuda")
    assert torch.equal(rank[end], w[end]) and torch.equal(root[end], succ[end])  # list ends keep theirs
    _holds(succ, w, root, torch.where(end, 0, rank))


@pytest.mark.parametrize("n", [14_336, 14_337, 30_011])
def test_weights_that_overflow_32_bits(kb, oracle_mod, n):
    rng = np.random.default_rng(n)
    succ = oracle_mod.gen_list(n, n, 0)
    w = np.full(n, 0xFFFFFFFF, np.uint32)
    w[rng.integers(0, n, n // 3)] = 0
    root_o, rank_o = oracle_mod.rank_list(succ, w)
    for mode in (1, 2):
        _, rank = kb.rank_list(dev64(succ), torch.from_numpy(w.view(np.int32)).cuda(),
                               tuning=kb.GpuTuning(level0_mode=mode, base_case_size=500))
        np.testing.assert_array_equal(host_i64(rank).view(np.uint64), rank_o)
