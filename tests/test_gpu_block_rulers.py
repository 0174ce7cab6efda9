"""Rulers placed by position and the one-CTA ranker, at the sizes where they
can go wrong: one element to past the one-CTA bound (16384), a last block that
its ruler falls out of, many lists, trees."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import dev32, dev64, host_i64, host_u64

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kb():
    import kascade_b200

    return kascade_b200


def _lists(n, parts, rng):
    succ = np.empty(n, np.uint64)
    cuts = np.sort(rng.choice(np.arange(1, n), size=parts - 1, replace=False)) if parts > 1 else []
    for seg in np.split(rng.permutation(n).astype(np.uint64), cuts):
        succ[seg[:-1]] = seg[1:]
        succ[seg[-1]] = seg[-1]
    return succ


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1024, 1025, 2047, 2049, 8191, 8193, 16383, 16384, 16385, 40961])
@pytest.mark.parametrize("parts", [1, 7, 2000])
def test_lists_around_the_one_cta_bounds(kb, oracle_mod, n, parts):
    rng = np.random.default_rng(n * 31 + parts)
    succ = _lists(n, min(parts, max(1, n // 2)), rng)
    w = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    root_o, rank_o = oracle_mod.rank_list(succ, w)
    for tuning in ({}, dict(ruler_spacing=3, base_case_size=700), dict(level0_mode=2, base_case_size=100)):
        root, rank = kb.rank_list(dev64(succ), dev32(w), tuning=kb.GpuTuning(**tuning))
        np.testing.assert_array_equal(host_u64(root), root_o)
        np.testing.assert_array_equal(host_u64(rank), rank_o)
    # in place, signed weights, roots keep their input
    s, k = succ.copy(), rng.integers(-(1 << 40), 1 << 40, n)
    s_o, k_o = s.copy(), k.copy()
    oracle_mod.local_pointer_chasing(s_o, k_o)
    sd, kd = dev64(s), dev64(k)
    kb.sparse_ruling_set(kb.SparseRulingSetConfig(), sd, kd)
    np.testing.assert_array_equal(host_u64(sd), s_o)
    np.testing.assert_array_equal(host_i64(kd), k_o)


@pytest.mark.parametrize("n", [3, 900, 1025, 8192])
def test_one_cta_ranks_trees(kb, oracle_mod, n):
    """Up to 8192 elements the list ranker takes any forest; above, two
    predecessors are an error."""
    par = oracle_mod.gen_forest(n, n, 0, 3 if n > 3 else 1)
    root_o, rank_o = oracle_mod.rank_list(par)
    root, rank = kb.rank_list(dev64(par))
    np.testing.assert_array_equal(host_u64(root), root_o)
    np.testing.assert_array_equal(host_u64(rank), rank_o)
    big = oracle_mod.gen_forest(n + 8192, n, 0, 1)
    with pytest.raises(kb.KascadeError) as e:
        kb.rank_list(dev64(big))
    assert e.value.name == "NOT_A_LIST"


@pytest.mark.parametrize("n", [9000, 70_001, 300_003])
def test_lists_that_meet_at_their_end(kb, oracle_mod, n):
    """Any number of lists may share their last element."""
    rng = np.random.default_rng(n)
    succ = _lists(n, 500, rng)
    ends = np.flatnonzero(succ == np.arange(n, dtype=np.uint64))
    succ[ends] = ends[0]
    root_o, rank_o = oracle_mod.rank_list(succ)
    for mode in (1, 2):
        root, rank = kb.rank_list(dev64(succ), tuning=kb.GpuTuning(level0_mode=mode))
        np.testing.assert_array_equal(host_u64(root), root_o)
        np.testing.assert_array_equal(host_u64(rank), rank_o)


@pytest.mark.parametrize("n,trees", [(1, 1), (3, 2), (8191, 5), (8193, 8193), (20_001, 3000), (300_007, 4)])
@pytest.mark.parametrize("tuning", [{}, dict(level0_mode=2, base_case_size=64), dict(ruler_spacing=3, base_case_size=5000)])
def test_tour_heads(kb, oracle_mod, n, trees, tuning):
    """Forests of one tree to more trees than the ranker keeps heads of (2048)."""
    par = oracle_mod.gen_forest(n, n + trees, 0, trees)
    root_o, depth_o = oracle_mod.root_forest(par)
    root, depth = kb.root_forest(dev64(par), tuning=kb.GpuTuning(**tuning))
    np.testing.assert_array_equal(host_u64(root), root_o)
    np.testing.assert_array_equal(host_u64(depth), depth_o)
