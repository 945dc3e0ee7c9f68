"""The domain sync's sort by the previous tree's leaves and the direct construction of the linked octree, against
numpy: the order must be the stable sort by SFC key whatever moved, the tree's arrays equal bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _keys(L, sim, pos):
    import torch
    dev = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in pos]
    keys = torch.zeros(pos[0].size, dtype=torch.int64, device="cuda")
    box = L.make_box((-0.5, 0.5) * 3, [1, 1, 1])
    torch.cuda.synchronize()
    L.check(sim.lib.sphb_compute_sfc_keys(*[L.ptr(d) for d in dev], L.ptr(keys), keys.numel(), C.byref(box), None),
            "keys")
    torch.cuda.synchronize()
    return keys.cpu().numpy().view(np.uint64)


MOVES = {
    "none": lambda p, rng: p,
    "small": lambda p, rng: p + rng.normal(0, 1e-4, p.shape),
    "cells": lambda p, rng: p + rng.normal(0, 2e-2, p.shape),
    "shuffled": lambda p, rng: p[:, rng.permutation(p.shape[1])],
    # more than 128 particles in one leaf: the radix sort
    "crowded": lambda p, rng: np.where(rng.random(p.shape[1]) < 0.2, 0.1 + 1e-3 * p, p),
    # pairs and triples at one point, and particles whose keys share their upper bits
    "equal keys": lambda p, rng: p[:, rng.integers(0, p.shape[1], p.shape[1])],
    "close keys": lambda p, rng: p[:, rng.integers(0, p.shape[1], p.shape[1])] + rng.uniform(0, 3e-6, p.shape),
}


@pytest.mark.parametrize("side", [4, 13, 32])
@pytest.mark.parametrize("move", sorted(MOVES))
def test_sync_orders_by_key(cuda_device, side, move):
    from sphexa_b200 import ic as icm
    from sphexa_b200 import lib as L
    from sphexa_b200.simulation import Simulation
    sim = Simulation(icm.sedov(side), "mixed")
    sim.sync()
    rng = np.random.default_rng(side)
    ids = sim.get("id")
    p = MOVES[move](np.stack([sim.get(f) for f in ("x", "y", "z")]), rng)
    p = p - np.round(p)
    for f, v in zip(("x", "y", "z"), p):
        sim.set(f, v)
    sim.sync()
    keys = _keys(L, sim, p)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(sim.get("id"), ids[order])
    assert np.array_equal(sim.keys(), keys[order])
    leaves, counts, layout = sim.tree()
    assert np.array_equal(layout, np.searchsorted(keys[order], leaves))
    assert np.array_equal(counts, np.diff(layout))


def _linked(leaves):
    """prefixes, child offsets, parents and level ranges of a cornerstone array, by sorting all ancestors"""
    level = (63 - np.log2(np.diff(leaves).astype(np.float64)).astype(np.int64)) // 3
    start = leaves[:-1]
    nodes = []
    for l in range(int(level.max()) + 1):
        s = start[level >= l]
        s = np.unique(s >> np.uint64(63 - 3 * l)) if l else np.zeros(1, np.uint64)
        nodes.append(s | np.uint64(1 << (3 * l)))
    prefixes = np.concatenate(nodes)
    counts = [len(q) for q in nodes]
    level_range = np.full(23, len(prefixes))
    level_range[:len(counts)] = np.concatenate([[0], np.cumsum(counts)[:-1]])
    child = np.zeros(len(prefixes), np.int64)
    parents = np.zeros(max(1, (len(prefixes) - 1) // 8), np.int64)
    leaf_prefix = {(int(s) >> (63 - 3 * int(l))) | (1 << (3 * int(l))) for s, l in zip(start, level)}
    for p, pre in enumerate(prefixes.tolist()):
        if pre in leaf_prefix:
            continue
        child[p] = np.searchsorted(prefixes, np.uint64(pre * 8))
        parents[(child[p] - 1) // 8] = p
    return prefixes, child, parents, level_range


@pytest.mark.parametrize("n,bucket", [(1, 8), (9, 8), (300, 1), (2000, 8), (5000, 5), (40_000, 1)])
def test_linked_octree(cuda_device, n, bucket):
    import torch
    from sphexa_b200 import lib as L
    lib = L.load()
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    keys[: n // 3] >>= np.uint64(20)
    keys = torch.from_numpy(np.sort(keys).view(np.int64)).cuda()
    cap = 40 * n + 4096
    leaves = torch.zeros(cap, dtype=torch.int64, device="cuda")
    counts = torch.zeros(cap, dtype=torch.int32, device="cuda")
    num = C.c_size_t()
    torch.cuda.synchronize()
    L.check(lib.sphb_compute_octree(L.ptr(keys), n, bucket, L.ptr(leaves), L.ptr(counts), cap, C.byref(num), None), "t")
    nl = num.value
    host = leaves[:nl + 1].cpu().numpy().view(np.uint64)
    k = keys.cpu().numpy().view(np.uint64)
    assert np.array_equal(counts[:nl].cpu().numpy(), np.diff(np.searchsorted(k, host)))
    nn = nl + (nl - 1) // 7
    prefixes = torch.zeros(nn, dtype=torch.int64, device="cuda")
    child = torch.zeros(nn, dtype=torch.int32, device="cuda")
    parents = torch.zeros(max(1, (nn - 1) // 8), dtype=torch.int32, device="cuda")
    i2l = torch.zeros(nn, dtype=torch.int32, device="cuda")
    l2i = torch.zeros(nn, dtype=torch.int32, device="cuda")
    level_range = (C.c_int * 23)()
    torch.cuda.synchronize()
    L.check(lib.sphb_build_octree(L.ptr(leaves), nl, L.ptr(prefixes), L.ptr(child), L.ptr(parents), level_range,
                                  L.ptr(i2l), L.ptr(l2i), None), "build")
    want = _linked(host)
    assert np.array_equal(prefixes.cpu().numpy().view(np.uint64), want[0])
    assert np.array_equal(child.cpu().numpy(), want[1])
    assert np.array_equal(parents.cpu().numpy(), want[2])
    assert np.array_equal(np.array(level_range[:]), want[3])
    # the two maps are inverse, leaves in key order
    i2l, l2i = i2l.cpu().numpy(), l2i.cpu().numpy()
    assert np.array_equal(np.sort(l2i), np.arange(nn))
    assert np.array_equal(i2l[l2i], np.arange(nn) - (nl - 1) // 7)


def _canonical(keys, bucket):
    """leaf starts of the cornerstone tree of sorted keys: a node with more than bucket keys splits, down to level 21"""
    leaves = []
    todo = [(0, 0, 0, len(keys))]
    while todo:
        start, level, a, b = todo.pop()
        if b - a <= bucket or level == 21:
            leaves.append(start)
            continue
        width = 1 << (63 - 3 * (level + 1))
        cuts = [start + d * width for d in range(9)]
        at = [a + int(np.searchsorted(keys[a:b], np.uint64(c))) for c in cuts[:8]] + [b]
        todo.extend((cuts[d], level + 1, at[d], at[d + 1]) for d in range(8))
    return np.array(sorted(leaves) + [1 << 63], dtype=np.uint64)


@pytest.mark.parametrize("bucket", [1, 8])
@pytest.mark.parametrize("kind", ["spread", "clustered", "equal", "deepest", "last"])
@pytest.mark.parametrize("n", [0, 1, 8, 9, 2049, 20_000])
def test_converged_leaves(cuda_device, n, kind, bucket):
    import torch
    from sphexa_b200 import lib as L
    lib = L.load()
    rng = np.random.default_rng(n)
    k = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    if kind == "clustered":
        k[: n // 2] >>= np.uint64(20)
    if kind == "equal":
        k[: n // 2] = np.uint64(0x123456789abcdef)
    if kind == "deepest":  # neighbouring cells of the deepest level
        k[: n // 2] = np.uint64(0x3fffffffffffffff) + rng.integers(0, 4, n // 2, dtype=np.uint64)
    if kind == "last":
        k[: n // 2] = np.uint64((1 << 63) - 1)
    k = np.sort(k)
    want = _canonical(k, bucket)
    keys = torch.from_numpy(k.view(np.int64)).cuda()
    cap = want.size + 7
    leaves = torch.full((cap,), -1, dtype=torch.int64, device="cuda")
    counts = torch.zeros(cap, dtype=torch.int32, device="cuda")
    num = C.c_size_t()
    torch.cuda.synchronize()
    L.check(lib.sphb_compute_octree(L.ptr(keys), n, bucket, L.ptr(leaves), L.ptr(counts), cap, C.byref(num), None), "t")
    assert num.value == want.size - 1
    assert np.array_equal(leaves.cpu().numpy()[:want.size].view(np.uint64), want)
    assert np.all(leaves.cpu().numpy()[want.size:] == -1)
    assert np.array_equal(counts.cpu().numpy()[:num.value], np.diff(np.searchsorted(k, want[:-1], "left"), append=n))
    # no room, or only the count asked for: the number of leaves all the same
    rc = lib.sphb_compute_octree(L.ptr(keys), n, bucket, L.ptr(leaves), L.ptr(counts), num.value, C.byref(num), None)
    assert rc == L.SPHB_ERR_CAPACITY and num.value == want.size - 1


@pytest.mark.parametrize("side", [4, 13, 27, 34, 36])
@pytest.mark.parametrize("move", ["cells", "crowded", "equal keys"])
def test_repeated_syncs_reach_the_converged_tree(cuda_device, side, move):
    """trees of up to and above the 2,048 leaves that single blocks update: splits, merges and forced leaves end at the
    tree in which a node with more than bucket_focus particles is split"""
    from sphexa_b200 import ic as icm
    from sphexa_b200 import lib as L
    from sphexa_b200.simulation import Simulation
    ic = icm.sedov(side)
    sim = Simulation(ic, "mixed")
    sim.sync()
    rng = np.random.default_rng(side)
    p = np.stack([sim.get(f) for f in ("x", "y", "z")])
    for f, v in zip(("x", "y", "z"), MOVES[move](p, rng)):
        sim.set(f, v - np.round(v))
    for _ in range(25):
        sim.sync()
    leaves, counts, layout = sim.tree()
    keys = sim.keys()
    assert np.array_equal(leaves, _canonical(keys, 64))
    assert np.array_equal(counts, np.diff(np.searchsorted(keys, leaves[:-1]), append=keys.size))
