"""Performance cases: list ranking and tree rooting as a program calls them.

Every case goes through the public entry points on device-resident arrays, the
form the library is built for: arrays in, (root, rank or depth) out.  The kinds
are the calls a user makes:

  list      rank_list: one array of lists in one call, unit or uint32 weights
  forest    root_forest: a parent array, roots and depths out
  batch     rank_batch: many lists and forests of uneven size in one call
  ruling    set_initial_ranking_state + sparse_ruling_set in place, the
            reference's own calling sequence
  doubling  set_initial_ranking_state + pointer_doubling in place on a forest

Inputs are made with plain torch from the seed: random list orders ("random"),
orders of runs of 64 consecutive indices joined by random jumps ("runs"),
random recursive trees ("rrt") and caterpillars whose spine is half of each
tree ("caterpillar"), vertices relabelled by a random permutation.
"""
import numpy as np
import torch

import kascade_b200 as kb

DEV = "cuda"


def listed():
    return [
        # the smallest request a service sees: one short list, latency only
        {"name": "list_1k", "kind": "list", "n": 1000, "layout": "random", "wbits": 0},
        # a mid-size weighted list of odd length
        {"name": "list_100k_w16", "kind": "list", "n": 100003, "layout": "random", "wbits": 16},
        # the plain configuration: 2^20 elements, unit weights
        {"name": "list_1m", "kind": "list", "n": 1 << 20, "layout": "random", "wbits": 0},
        # an order with locality, full-range weights, ragged length
        {"name": "list_20m_runs_w32", "kind": "list", "n": 20000003, "layout": "runs", "wbits": 32},
        # the headline: 2^28 elements in random order, weights below 2^16
        {"name": "list_268m_w16", "kind": "list", "n": 1 << 28, "layout": "random", "wbits": 16},
        # a small hierarchy rooted on its own: deep trees, odd size
        {"name": "forest_50k_cat", "kind": "forest", "n": 50021, "shape": "caterpillar", "trees": 4},
        # an ordinary forest of shallow random trees
        {"name": "forest_4m_rrt", "kind": "forest", "n": 4194301, "shape": "rrt", "trees": 64},
        # the large rooting configuration: 64 caterpillars over 2^26 vertices
        {"name": "forest_67m_cat", "kind": "forest", "n": 1 << 26, "shape": "caterpillar", "trees": 64},
        # what a serving lane collects at once: requests of 2^8 .. 2^18 elements
        {"name": "batch_128_3m", "kind": "batch", "count": 128, "lo": 8, "hi": 18, "total": 3000017, "wbits": 16},
        # the batched configuration: 4096 instances of 2^6 .. 2^22, 2^28 elements
        {"name": "batch_4096_268m", "kind": "batch", "count": 4096, "lo": 6, "hi": 22, "total": 1 << 28, "wbits": 16},
        # the reference-shaped in-place call on a large list
        {"name": "ruling_6m", "kind": "ruling", "n": 6000011, "layout": "random"},
        # the reference-shaped pointer doubling, which takes any forest
        {"name": "doubling_1m_cat", "kind": "doubling", "n": 1000003, "shape": "caterpillar", "trees": 16},
    ]


def _log_uniform(rng, lo, hi):
    """An odd-leaning size, uniform over its logarithm in [2^lo, 2^hi]."""
    return int(2.0 ** rng.uniform(lo, hi)) | rng.randrange(2)


def draw(rng):
    kind = rng.choice(["list", "list", "list", "forest", "forest", "batch", "batch", "ruling", "doubling"])
    if kind == "list":
        return {"kind": kind, "n": _log_uniform(rng, 6, 27.9), "layout": rng.choice(["random", "random", "runs"]),
                "wbits": rng.choice([0, 16, 16, 32])}
    if kind == "forest":
        n = _log_uniform(rng, 6, 25.9)
        return {"kind": kind, "n": n, "shape": rng.choice(["rrt", "rrt", "caterpillar"]),
                "trees": min(rng.choice([1, 4, 64]), n // 16)}
    if kind == "batch":
        lo, total = rng.randrange(6, 9), _log_uniform(rng, 16, 27.9)
        count = min(int(2.0 ** rng.uniform(4, 12)), total >> (lo + 1))
        return {"kind": kind, "count": count, "lo": lo, "hi": lo + rng.randrange(8, 15), "total": total,
                "wbits": rng.choice([0, 16, 16, 32])}
    if kind == "ruling":
        return {"kind": kind, "n": _log_uniform(rng, 6, 27), "layout": rng.choice(["random", "random", "runs"])}
    n = _log_uniform(rng, 6, 24)
    return {"kind": kind, "n": n, "shape": rng.choice(["rrt", "caterpillar"]), "trees": min(rng.choice([1, 16]), n // 16)}


def _rand(n, gen):
    return torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)


def _instances(case):
    """Sizes (log-uniform, rescaled to the total) and kinds (70% lists, 30%
    forests) of a batch's instances."""
    rng = np.random.default_rng(case["count"] * 1000003 + case["total"])
    raw = 2.0 ** rng.uniform(case["lo"], case["hi"], case["count"])
    sizes = np.maximum((raw * (case["total"] / raw.sum())).astype(np.int64), 16)
    sizes[np.argmax(sizes)] += case["total"] - sizes.sum()
    kinds = np.where(rng.random(case["count"]) < 0.7, kb.SEG_LIST, kb.SEG_FOREST)
    return sizes, kinds


def _orders(sizes, gen):
    """Random orders of every instance: positions 0..total-1, each instance's
    range shuffled in itself."""
    total = int(sizes.sum())
    if len(sizes) == 1:
        return torch.randperm(total, generator=gen, device=DEV)
    seg = torch.repeat_interleave(torch.arange(len(sizes), device=DEV), torch.from_numpy(sizes).to(DEV))
    key = (seg << 44) | torch.randint(1 << 44, (total,), generator=gen, device=DEV)
    return torch.argsort(key)


def _list(case, gen):
    n = case["n"]
    if case["layout"] == "random":
        order = torch.randperm(n, generator=gen, device=DEV)
    else:
        runs = (n + 63) // 64
        order = (torch.randperm(runs, generator=gen, device=DEV)[:, None] * 64
                 + torch.arange(64, device=DEV)[None, :]).flatten()
        order = order[order < n]
    succ = torch.empty_like(order)
    succ[order[:-1]] = order[1:]
    succ[order[-1]] = order[-1]
    return succ


def _parents(n, shape, trees, gen):
    """Parents of positions 0..n-1 before relabelling: `trees` equal blocks,
    each rooted at its first position."""
    pos = torch.arange(n, device=DEV)
    size = -(-n // trees)
    base = pos // size * size
    at = pos - base
    u = _rand(n, gen)
    if shape == "rrt":
        return base + torch.clamp((u * at).long(), max=n).minimum(torch.clamp(at - 1, min=0))
    spine = max(1, size // 2)
    leaf = torch.clamp((u * spine).long(), max=spine - 1)
    return base + torch.where(at < spine, torch.clamp(at - 1, min=0), leaf)


def _forest(case, gen):
    par = _parents(case["n"], case["shape"], case["trees"], gen)
    order = torch.randperm(case["n"], generator=gen, device=DEV)
    out = torch.empty_like(par)
    out[order] = order[par]
    return out


def _batch(case, gen):
    """Concatenated instances with instance-local indices: random lists and
    random recursive trees (one tree per 2^16 vertices, at least one)."""
    sizes, kinds = _instances(case)
    order = _orders(sizes, gen)
    total = case["total"]
    size_d = torch.from_numpy(sizes).to(DEV)
    off = torch.repeat_interleave(torch.cumsum(size_d, 0) - size_d, size_d)
    size = torch.repeat_interleave(size_d, size_d)
    forest = torch.repeat_interleave(torch.from_numpy((kinds == kb.SEG_FOREST)).to(DEV), size_d)
    pos = torch.arange(total, device=DEV)
    at = pos - off
    # lists: the next position, the last one pointing to itself
    nxt = torch.where(at + 1 < size, pos + 1, pos)
    # forests: a uniform earlier position of the same tree
    tree = (size + torch.clamp(size >> 16, min=1) - 1) // torch.clamp(size >> 16, min=1)
    start = at // tree * tree
    j = at - start
    par = off + start + torch.clamp((_rand(total, gen) * j).long(), max=total).minimum(torch.clamp(j - 1, min=0))
    nxt = torch.where(forest, par, nxt)
    del par, size, forest, at, start, j, tree, pos
    out = torch.empty_like(order)
    out[order] = order[nxt] - off
    return out, sizes, kinds


def _weights(n, wbits, gen):
    if not wbits:
        return None
    return torch.randint(1 << wbits, (n,), generator=gen, device=DEV, dtype=torch.int64).to(torch.int32)


def _inputs(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind in ("list", "ruling"):
        data = {"succ": _list(case, gen)}
    elif kind in ("forest", "doubling"):
        data = {"succ": _forest(case, gen)}
    else:
        succ, sizes, kinds = _batch(case, gen)
        data = {"succ": succ, "sizes": sizes, "kinds": kinds}
    data["weights"] = _weights(data["succ"].numel(), case.get("wbits", 0), gen)
    return data


def prepare(case, seed):
    state = _inputs(case, seed)
    state["kind"] = case["kind"]
    if case["kind"] == "batch":
        state["segments"] = kb.make_segments(state["sizes"], state["kinds"])
    return state


def run(state):
    kind, succ = state["kind"], state["succ"]
    if kind == "list":
        return kb.rank_list(succ, state["weights"])
    if kind == "forest":
        return kb.root_forest(succ)
    if kind == "batch":
        return kb.rank_batch(succ, state["segments"], state["weights"])
    root, rank = kb.set_initial_ranking_state(succ)
    if kind == "ruling":
        kb.sparse_ruling_set(kb.SparseRulingSetConfig(), root, rank)
    else:
        kb.pointer_doubling(kb.PointerDoublingConfig(), root, rank)
    return root, rank


def work(case):
    """Indices (and weights) read once, root and rank written once."""
    n = case["total"] if case["kind"] == "batch" else case["n"]
    return {"bytes": n * (24 + (4 if case.get("wbits", 0) else 0)), "flops": 0}


def exact(case, seed):
    """Roots and ranks by pointer jumping in plain torch, 64-bit integers."""
    data = _inputs(case, seed)
    succ = data["succ"]
    n = succ.numel()
    off = None
    if case["kind"] == "batch":
        size = torch.from_numpy(data["sizes"]).to(DEV)
        off = torch.repeat_interleave(torch.cumsum(size, 0) - size, size)
        succ = succ + off
    step = torch.ones(n, dtype=torch.int64, device=DEV)
    if data["weights"] is not None:
        step = data["weights"].long() & 0xFFFFFFFF
        if off is not None:  # a batch's forests report depths
            forest = torch.from_numpy(data["kinds"] == kb.SEG_FOREST).to(DEV)
            step = torch.where(torch.repeat_interleave(forest, size), 1, step)
    pos = torch.arange(n, device=DEV)
    rank = torch.where(succ == pos, 0, step)
    del step, pos
    while True:
        nxt = succ[succ]
        if torch.equal(nxt, succ):
            break
        rank = rank + rank[succ]
        succ = nxt
    return succ if off is None else succ - off, rank
