"""The pair loops where their branches meet: density contrasts on all three branches of the Atwood weights, particles
at the same position, and particle counts around the edges of a group of 32 and of a block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("xm", "kx", "gradh", "prho", "c", "c11", "c12", "c13", "c22", "c23", "c33", "divv", "curlv", "ax", "ay", "az",
          "du", "alpha")


def contrast(side, keep=None, coincident=0, seed=5):
    """A jittered lattice with random velocities and masses between m and 1.8 m, so that the densities of a pair differ
    by anything from 0 to 30 %; the last `coincident` particles sit on the first ones."""
    from sphexa_b200 import ic as icm
    f = icm.sedov(side, seed=seed)
    rng = np.random.default_rng(seed)
    n = f["x"].size if keep is None else keep
    pick = np.sort(rng.permutation(f["x"].size)[:n])
    for k in icm.CONSERVED_FIELDS:
        f[k] = f[k][pick].copy()
    f["id"] = np.arange(n, dtype=np.uint64)
    smooth = 1.0 + 0.4 * np.sin(2.0 * np.pi * f["x"])
    f["m"] = f["m"] * smooth * rng.uniform(1.0, 1.3, n)
    f["h"] = f["h"] * (f["x"].size / n) ** (1.0 / 3.0) * rng.uniform(0.95, 1.05, n)
    for k in ("vx", "vy", "vz"):
        f[k] = rng.uniform(-1.0, 1.0, n)
    f["temp"] = f["temp"].max() * rng.uniform(0.5, 1.0, n)
    f["alpha"] = rng.uniform(0.05, 1.0, n)
    for q in range(coincident):
        for k in ("x", "y", "z"):
            f[k][n - 1 - q] = f[k][q]
    return f


@pytest.mark.parametrize("side,keep,coincident", [(8, None, 0), (8, 481, 0), (9, 720, 3), (13, 2177, 0), (13, None, 5)])
def test_fp64_forces_against_the_restatement(cuda_device, side, keep, coincident):
    """One force computation against the C restatement, which sums neighbour by neighbour; the pair loops sum eight at a
    time and add the partial sums. A term's rounding differs by a few 1e-16 (reciprocals for divisions). Either order of
    100 additions is off by at most sqrt(100) of that for rounding errors that are independent, and divv, curlv, du and
    the accelerations are differences of larger terms: 1e-12 of a field's largest magnitude leaves a factor 100."""
    from oracle import restated
    from sphexa_b200.simulation import Simulation
    ic = contrast(side, keep, coincident)
    g = Simulation(ic, "fp64")
    o = restated.OracleSim(ic)
    g.compute_forces()
    o.compute_forces()
    assert np.array_equal(g.get("nc"), o.get("nc"))
    for f in FIELDS:
        a, b = g.get(f), o.get(f)
        assert np.all(np.isfinite(a)), f
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b)), f


@pytest.mark.parametrize("precision,av_clean", [("mixed", False), ("fp64", False), ("mixed", True)])
@pytest.mark.parametrize("n", [1, 31, 33, 16384, 16385, 65536, 65537])
def test_lanes_per_target_leave_the_sums_alone(cuda_device, n, precision, av_clean):
    """Eight, four or one lane share a target by the number of targets; an ensemble's launches always use one. The same
    particles give the same bits on both sides of either limit."""
    from sphexa_b200.ensemble import Ensemble
    from sphexa_b200.simulation import Simulation
    ic = contrast(max(8, int(np.ceil(n ** (1.0 / 3.0)))), n)
    ic["params"]["avClean"] = av_clean
    sim, ens = Simulation(ic, precision), Ensemble([ic], precision)
    sim.step()
    ens.step(1, graph=False)
    for f in FIELDS + ("x", "vx", "temp", "nc"):
        assert np.array_equal(sim.get(f), ens.get(0, f), equal_nan=True), f
