"""Neighbour searches with one, four and eight lanes per target: the lists against a k-d tree, and listed searches against
the full ones, on both sides of the sizes and of the list length at which the number of lanes changes."""
import numpy as np
import pytest

from test_gpu_skin import _pair, _run, _stirred
from test_gpu_skin_build import clumps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,spread,ngmax", [(9, 1.0, 150), (33, 1.0, 150), (263, 0.5, 150), (4099, 0.3, 150),
                                            (4100, 0.3, 20), (10_000, 0.3, 150), (10_001, 0.3, 150),
                                            (40_000, 0.3, 150), (40_001, 0.3, 150)])
def test_lists_match_a_kd_tree(cuda_device, n, spread, ngmax, precision):
    from scipy.spatial import cKDTree
    from sphexa_b200.simulation import Simulation
    f = clumps(n, 5, spread)
    f["params"]["nbSkin"] = 0.0
    f["params"]["ngmax"] = ngmax
    f["params"]["ng0"] = min(f["params"]["ng0"], ngmax - 10)
    if ngmax == 20:  # a clump that no smoothing length of the iteration brings below ngmax
        rng = np.random.default_rng(1)
        for k in ("x", "y", "z"):
            f[k][100:160] = 0.1 + rng.uniform(0, 1e-7, 60)
    sim = Simulation(f, precision)
    sim.compute_forces()
    p = np.stack([sim.get(k) for k in ("x", "y", "z")], 1)
    h, nc, lists = sim.get("h"), sim.get("nc").astype(np.int64), sim.neighbors()
    tree = cKDTree((p + 0.5) % 1.0, boxsize=1.0)
    near = tree.query_ball_point((p + 0.5) % 1.0, np.minimum(2 * h * (1 + 1e-9), 0.49999), workers=4)
    over = 0
    for i in range(n):
        if 2 * h[i] > 0.49:
            continue  # beyond the k-d tree's periodic range
        j = np.sort(np.array(near[i]))
        j = j[j != i]
        d = p[j] - p[i]
        d -= np.round(d)
        d2 = (d * d).sum(1)
        edge = np.abs(d2 - 4 * h[i] ** 2) < 1e-12 * h[i] ** 2
        want = j[(d2 < 4 * h[i] ** 2)]
        if edge.any():
            continue  # decided by the last bit
        assert nc[i] == want.size + 1, i
        got = lists[i][: min(want.size, ngmax)]
        assert np.array_equal(got, want[:ngmax]), i
        over += want.size > ngmax
    if ngmax == 20:
        assert over > 0  # truncated lists are among the tested


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("side", [40, 66, 68])
def test_listed_searches(cuda_device, side, precision):
    a, b = _pair(_stirred(side, radius=0.15, speed=40.0), precision)
    _run(a, b, 4)
    assert a.search_stats()["deferred_groups"] > 0


def test_lists_on_both_sides_of_the_limit(cuda_device):
    """a stirred region that spreads: few of its groups are listed first, then more than those that take eight lanes"""
    a, b = _pair(_stirred(80, radius=0.173), "mixed")
    lengths = []
    for _ in range(7):
        before = a.search_stats()["deferred_groups"]
        _run(a, b, 1)
        lengths.append(a.search_stats()["deferred_groups"] - before)
    assert any(0 < n <= 1500 for n in lengths) and max(lengths) > 1500, lengths


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [10_000, 10_001, 40_000, 40_001])
def test_row_builds(cuda_device, n, precision):
    a, b = _pair(clumps(n, 5, 0.5), precision)
    _run(a, b, 3)
    assert a.search_stats()["skin_builds"] >= 1
