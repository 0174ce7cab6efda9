"""Ranking in-trees by contracting their paths: tree rooting and the
pointer-doubling entry points, around the sizes at which levels are added, on
shapes from a star to one path, against pointer jumping in numpy (integers:
the results are equal)."""
from __future__ import annotations

import numpy as np
import pytest

import torch

from gpu_util import dev64, host_i64

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kb():
    import kascade_b200

    return kascade_b200


def _shapes(n, rng):
    order = rng.permutation(n)
    star = np.full(n, order[0], np.int64)
    path = np.empty(n, np.int64)
    path[order[1:]] = order[:-1]
    path[order[0]] = order[0]
    attach = np.empty(n, np.int64)  # random recursive trees, seven of them
    at = np.arange(n)
    up = np.minimum((rng.random(n) * at).astype(np.int64), np.maximum(at - 1, 0))
    up[:7] = at[:7]
    attach[order] = order[up]
    comb = np.empty(n, np.int64)  # a path over half the elements, the rest leaves of it
    half = max(1, n // 2)
    up = np.where(at < half, np.maximum(at - 1, 0), rng.integers(0, half, n))
    comb[order] = order[up]
    return {"star": star, "path": path, "attach": attach, "comb": comb, "roots": np.arange(n)}


def _jump(succ, w):
    succ, d = succ.copy(), np.where(succ == np.arange(len(succ)), 0, w).astype(np.int64)
    while True:
        nxt = succ[succ]
        if np.array_equal(nxt, succ):
            return succ, d
        d = d + d[succ]
        succ = nxt


@pytest.mark.parametrize("n", [1, 2, 33, 4095, 4096, 4097, 12_289, 70_001, 1_000_003])
def test_shapes_and_sizes(kb, n):
    rng = np.random.default_rng(n)
    w = rng.integers(-(1 << 40), 1 << 40, n)
    for name, succ in _shapes(n, rng).items():
        root_o, depth_o = _jump(succ, np.ones(n, np.int64))
        for t in ({}, dict(ruler_spacing=2, ruler_spacing_deep=7, base_case_size=100), dict(ruler_spacing=50)):
            root, depth = kb.root_forest(dev64(succ.astype(np.uint64)), tuning=kb.GpuTuning(**t))
            np.testing.assert_array_equal(host_i64(root), root_o, err_msg=name)
            np.testing.assert_array_equal(host_i64(depth), depth_o, err_msg=name)
        s, r = dev64(succ.astype(np.uint64)), dev64(np.ones(n, np.int64).view(np.uint64))
        kb.rank_via_euler_tour(kb.EulerTourConfig(), s, r)
        isroot = succ == np.arange(n)
        np.testing.assert_array_equal(host_i64(s), root_o, err_msg=name)
        np.testing.assert_array_equal(host_i64(r), np.where(isroot, 1, depth_o), err_msg=name)  # roots keep theirs
        _, rank_o = _jump(succ, w)
        s, r = dev64(succ.astype(np.uint64)), dev64(w.view(np.uint64))
        kb.pointer_doubling(kb.PointerDoublingConfig(), s, r)
        np.testing.assert_array_equal(host_i64(s), root_o, err_msg=name)
        np.testing.assert_array_equal(host_i64(r), np.where(isroot, w, rank_o), err_msg=name)


@pytest.mark.parametrize("n", [2000, 30_000, 500_000])
def test_cycles_are_reported(kb, n):
    rng = np.random.default_rng(n)
    order = rng.permutation(n)
    pairs = np.empty(n, np.int64)  # two-element cycles: most hold no ruler
    pairs[order[0::2]], pairs[order[1::2]] = order[1::2], order[0::2]
    tail = _shapes(n, rng)["path"]  # a path into a three-element cycle
    end = np.flatnonzero(tail == np.arange(n))[0]
    up = {v: u for u, v in enumerate(tail) if u != v}
    tail[end] = up[up[end]]
    ring = np.empty(n, np.int64)
    ring[order] = np.roll(order, 1)
    for succ in (pairs, tail, ring):
        for run in (lambda s: kb.root_forest(s), lambda s: kb.rank_list(s, algorithm=kb.Algorithm.PointerDoubling)):
            with pytest.raises(kb.KascadeError) as e:
                run(dev64(succ.astype(np.uint64)))
            assert e.value.name == "CYCLE"


@pytest.mark.parametrize("n", [1 << 26, (1 << 26) + 1, (1 << 26) + 70_001])
@pytest.mark.parametrize("hubs", [0, 50_000])
def test_both_kinds_of_child_flags(kb, n, hubs):
    """Child flags in bytes and in bits: depth and root follow the parent's."""
    if hubs:
        g = torch.Generator(device="cuda")
        g.manual_seed(n)
        par = torch.randint(0, hubs, (n,), device="cuda", generator=g)
        par[:hubs] = (torch.arange(hubs, device="cuda") - 1).clamp(min=0)  # the hubs: one path
    else:
        par = kb.gen_forest(n, n, 0, 3, 0)
    root, depth = kb.root_forest(par)
    idx = torch.arange(n, device="cuda")
    top = par == idx
    assert bool((depth == torch.where(top, 0, depth[par] + 1)).all())
    assert bool((root == torch.where(top, idx, root[par])).all())


def test_bits_in_a_batch(kb):
    n = (1 << 27) + 5
    par = kb.gen_forest(n, 9, 0, 2, 0)
    segs = kb.make_segments(np.array([n], np.int64), np.array([kb.SEG_FOREST], np.int64))
    root, depth = kb.rank_batch(par, segs)
    root_f, depth_f = kb.root_forest(par)
    assert torch.equal(root, root_f) and torch.equal(depth, depth_f)
