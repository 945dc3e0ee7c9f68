"""Row builds: the lists of a build step come from the rows themselves, and the rows' build distances from FP32 pair
distances where the group is compact, from FP64 ones where it reaches far (stray particles between clumps)."""
import numpy as np
import pytest

from test_gpu_skin import _pair, _run

pytestmark = pytest.mark.gpu


def clumps(n, seed, spread):
    """n particles of the Sedov lattice, most of them drawn towards eight points, some left where they were: groups of
    32 that hold both reach several search radii. The smoothing lengths are off, so that the first step iterates h."""
    from sphexa_b200 import ic as icm
    side = int(np.ceil(n ** (1.0 / 3.0)))
    f = icm.sedov(side, seed=seed)
    rng = np.random.default_rng(seed)
    pick = np.sort(rng.permutation(f["x"].size)[:n])
    for k in icm.CONSERVED_FIELDS:
        f[k] = f[k][pick].copy()
    f["id"] = np.arange(n, dtype=np.uint64)
    drawn = rng.random(n) < 0.9
    for k in ("x", "y", "z"):
        to = np.where(f[k] < 0, -0.25, 0.25)
        f[k] = np.where(drawn, to + (f[k] - to) * spread, f[k])
        f["v" + k] = rng.uniform(-0.2, 0.2, n)
    f["h"] = np.where(drawn, f["h"] * spread, f["h"]) * rng.uniform(0.6, 1.3, n)
    f["temp"] = np.full(n, f["temp"].min())
    f["params"]["minDt"] = f["params"]["minDt_m1"] = 1e-4
    return f


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,spread", [(65, 1.0), (1000, 0.5), (4097, 0.3), (9000, 0.25)])
def test_lists_of_build_and_refilter_steps(cuda_device, precision, n, spread):
    a, b = _pair(clumps(n, 3, spread), precision)
    _run(a, b, 4)
    assert a.search_stats()["skin_builds"] >= 1
