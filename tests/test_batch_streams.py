"""Where a batch's forests run beside its lists: on a second stream of the
caller's priority, or on the caller's own where that belongs to an SM
partition."""
from __future__ import annotations

import ctypes

import pytest

import fake_runtime as fr

U64, P = ctypes.c_uint64, ctypes.c_void_p


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fr.load(tmp_path_factory.mktemp("fake"))


@pytest.fixture()
def ctx(lib):
    h = P()
    assert lib.kascade_ctx_create(0, ctypes.byref(h)) == 0
    yield h
    assert lib.kascade_ctx_destroy(h) == 0


def _batch(lib, ctx, stream):
    segs, total = fr.segments([100_000, 30_000], [0, 1])
    lib.fake_reset(ctypes.c_size_t(-1).value)
    at = fr.DEVICE
    st = lib.kascade_rank_batch(ctx, segs, 2, P(at), None, U64(total), P(at + (1 << 30)), P(at + (2 << 30)), None,
                                P(stream))
    assert st == 0
    rows = fr.launches(lib)
    assert any("k_tree_leaves" in k for k, _ in rows) and any("k_propagate" in k for k, _ in rows)
    return {s for k, s in rows if "k_tree" in k}, {s for k, s in rows if "k_chase" in k or "k_propagate" in k}


def test_priority_follows_the_callers_stream(lib, ctx):
    held = lib.fake_streams()
    for priority in (-5, -5, 0, -3, -5):
        s = lib.fake_stream(priority, 0)
        forests, lists = _batch(lib, ctx, s)
        assert lists == {s} and len(forests) == 1
        side = forests.pop()
        assert side != s and lib.fake_priority(side) == priority
        held += 1
        assert lib.fake_streams() == held + 1  # the caller's so far, and one second stream


def test_default_stream(lib, ctx):
    forests, lists = _batch(lib, ctx, 0)
    assert lists == {0} and lib.fake_priority(forests.pop()) == 0


def test_a_partitions_stream_keeps_all_work(lib, ctx):
    s = lib.fake_stream(-1, 1)
    assert _batch(lib, ctx, s) == ({s}, {s})
    plain = lib.fake_stream(-1, 0)
    forests, _ = _batch(lib, ctx, plain)
    assert forests != {plain}


def test_a_context_with_a_budget_keeps_one_stream(lib, ctx):
    s = lib.fake_stream(0, 0)
    assert lib.kascade_ctx_set_sm_budget(ctx, 100) == 0
    assert _batch(lib, ctx, s) == ({s}, {s})
