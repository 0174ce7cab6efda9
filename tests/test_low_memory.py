"""Calls whose memory does not suffice for the write-free level 0 stamp instead:
what ran when large lists still stamped by size runs as before.  The host code
allocates from a device of settable size; its launches show the path taken."""
from __future__ import annotations

import ctypes

import pytest

import fake_runtime as fr

U64, P = ctypes.c_uint64, ctypes.c_void_p
OOM = 6
MIB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fr.load(tmp_path_factory.mktemp("fake"))


@pytest.fixture()
def ctx(lib):
    h, before = P(), lib.fake_used()
    assert lib.kascade_ctx_create(0, ctypes.byref(h)) == 0
    yield h
    assert lib.kascade_ctx_destroy(h) == 0
    assert lib.fake_used() == before


def _paths(lib):
    names = [k for k, _ in fr.launches(lib)]
    return any("k_chase_log" in k for k in names), any("k_place" in k for k in names)


def _ruling(lib, ctx, n, **o):
    return lib.kascade_sparse_ruling_set(ctx, ctypes.byref(fr.opts(lib, **o)), P(fr.DEVICE), P(fr.DEVICE + (1 << 40)),
                                         U64(n), P(0))


def _list(lib, ctx, n, **o):
    return lib.kascade_rank_list(ctx, P(fr.DEVICE), P(fr.DEVICE + (1 << 39)), U64(n), P(fr.DEVICE + (1 << 40)),
                                 P(fr.DEVICE + (2 << 40)), ctypes.byref(fr.opts(lib, **o)), P(0))


@pytest.mark.parametrize("call,n,need", [(_ruling, 1 << 25, 22), (_ruling, 1 << 28, 22), (_list, 1 << 24, 25),
                                         (_list, 1 << 28, 25)])
@pytest.mark.parametrize("mode", [0, 2])
def test_memory_for_stamps_only(lib, ctx, call, n, need, mode):
    """`need`: the bytes an element that the call took when its lists stamped."""
    lib.fake_reset(n * need + 64 * MIB)
    assert call(lib, ctx, n, level0_mode=mode) == 0
    assert _paths(lib) == (False, False)
    lib.fake_reset(ctypes.c_size_t(-1).value)  # the memory is there: write-free
    assert call(lib, ctx, n, level0_mode=mode) == 0
    assert _paths(lib) == (True, True)


@pytest.mark.parametrize("call,n,need", [("kascade_pointer_doubling", 1 << 28, 52.3),
                                         ("kascade_pointer_doubling", (1 << 31) + 7, 52.3),
                                         ("kascade_root_forest", 1 << 28, 39)])
def test_trees(lib, ctx, call, n, need):
    """Pointer doubling took 52 bytes an element by rounds, rooting far more by its tour."""
    lib.fake_reset(int(n * need))
    a = [P(fr.DEVICE + (k << 40)) for k in range(3)]
    if call == "kascade_root_forest":
        assert lib.kascade_root_forest(ctx, a[0], U64(n), a[1], a[2], None, P(0)) == 0
    else:
        assert lib.kascade_pointer_doubling(ctx, None, a[0], a[1], U64(n), P(0)) == 0


def test_memory_for_nothing(lib, ctx):
    lib.fake_reset(10 << 25)
    assert _ruling(lib, ctx, 1 << 25) == OOM
    assert not fr.launches(lib) and lib.fake_used() <= 4096
    lib.fake_reset(ctypes.c_size_t(-1).value)
    assert _ruling(lib, ctx, 1 << 25) == 0


def test_the_largest_in_place_list(lib, ctx):
    """2^32 - 2 elements beside the caller's 16 bytes an element on 180 GB."""
    n = (1 << 32) - 2
    lib.fake_reset(180 * 10 ** 9 - 16 * n)
    assert _ruling(lib, ctx, n) == 0
    assert _paths(lib) == (False, False)


@pytest.mark.parametrize("fixed", [False, True])
def test_batch(lib, ctx, fixed):
    """Lists give way for the forests' memory too; a plan's capture takes the
    path of its first run and allocates nothing."""
    nl, nf = 20_000_000, 10_000_000
    segs, total = fr.segments([nl, nf], [0, 1])
    a = [P(fr.DEVICE + (k << 38)) for k in range(3)]
    lib.fake_reset(25 * nl + 50 * nf + 128 * MIB)
    if fixed:
        plan = P()
        st = lib.kascade_batch_plan_create(0, segs, 2, a[0], None, U64(total), a[1], a[2], None, ctypes.byref(plan))
        assert st == 0 and lib.fake_grown_in_capture() == 0
        assert sum("k_batch_prepare" in k for k, _ in fr.launches(lib)) == 2
        assert lib.kascade_batch_plan_destroy(plan) == 0
    else:
        assert lib.kascade_rank_batch(ctx, segs, 2, a[0], None, U64(total), a[1], a[2], None, P(0)) == 0
    assert _paths(lib) == (False, False)
    assert any("k_tree_leaves" in k for k, _ in fr.launches(lib))


def test_plan_with_memory(lib):
    segs, total = fr.segments([20_000_000, 100_000], [0, 1])
    a = [P(fr.DEVICE + (k << 38)) for k in range(3)]
    lib.fake_reset(ctypes.c_size_t(-1).value)
    plan = P()
    assert lib.kascade_batch_plan_create(0, segs, 2, a[0], None, U64(total), a[1], a[2], None, ctypes.byref(plan)) == 0
    assert sum("k_chase_log" in k for k, _ in fr.launches(lib)) == 2 and lib.fake_grown_in_capture() == 0
    assert lib.kascade_batch_plan_destroy(plan) == 0
