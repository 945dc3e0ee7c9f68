"""The ensemble's sort where its trees no longer fit: a member whose particles crowd into leaves of the last rebuild past
what a warp sorts, and trees of large buckets, against single simulations bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "h", "temp", "vx", "vy", "vz", "du_m1", "alpha", "id", "keys", "nc")


def contracting(side, seed):
    """cold gas falling towards the middle of an octant's octant, the density growing by up to 6 % a step"""
    from sphexa_b200 import ic as icm
    f = icm.sedov(side, seed=seed)
    dt = 0.01
    d = {a: f[a] - 0.125 for a in "xyz"}
    inside = d["x"] ** 2 + d["y"] ** 2 + d["z"] ** 2 < 0.3 ** 2
    for a in "xyz":
        f["v" + a] = np.where(inside, -4.0 * d[a], 0.0)
        f[a + "_m1"] = f["v" + a] * dt
    f["temp"] = np.full(f["x"].size, f["temp"].min())
    f["params"].update(minDt=dt, minDt_m1=dt)
    return f


def compare(ics, steps, graph, precision):
    from sphexa_b200.ensemble import Ensemble
    from sphexa_b200.simulation import Simulation
    ens = Ensemble(ics, precision)
    sims = [Simulation(ic, precision) for ic in ics]
    leaves = [sim.tree()[0] for sim in sims]
    ens.step(steps, graph=graph)
    for k, sim in enumerate(sims):
        for _ in range(steps):
            sim.step()
        for f in FIELDS:
            assert np.array_equal(ens.get(k, f), sim.keys() if f == "keys" else sim.get(f)), (k, f)
    return [int(np.diff(np.searchsorted(ens.get(k, "keys"), l)).max()) for k, l in enumerate(leaves)]


@pytest.mark.parametrize("graph,precision,steps", [(True, "mixed", 30), (False, "mixed", 25), (True, "fp64", 25)])
def test_a_leaf_of_one_member_outgrows_a_warp(cuda_device, graph, precision, steps):
    from sphexa_b200 import ic as icm
    largest = compare([icm.sedov(12, seed=1), contracting(29, 2), icm.sedov(9, seed=3)], steps, graph, precision)
    assert max(largest[0], largest[2]) <= 128 < largest[1] <= 2048


@pytest.mark.parametrize("bucket,side,graph", [(65, 29, True), (300, 26, True), (1024, 40, True), (1024, 40, False),
                                               (1025, 40, True)])
def test_trees_of_large_buckets(cuda_device, bucket, side, graph, monkeypatch):
    """up to a leaf past 2,048 particles, in a captured step and in an eager one, and buckets that no leaf sort takes"""
    from sphexa_b200 import ic as icm
    from sphexa_b200 import lib as L
    plain = L.make_params
    monkeypatch.setattr(L, "make_params", lambda p, precision: plain(p, precision, bucket))
    largest = compare([contracting(side, 2), icm.sedov(13, seed=3)], 25 if bucket < 1024 else 50, graph, "mixed")
    assert (max(largest) > 2048) == (bucket >= 1024)
    assert max(largest) > 128
