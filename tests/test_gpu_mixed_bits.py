"""The mixed form's bits. The AV switches jump where divv changes its sign, so a last bit of an FP32 sum moves alpha of
such a particle by its full range, and an unstable flow amplifies it: the order of every FP32 sum and FMA is part of the
results. The digests were recorded with one lane per target and the compiler's own contraction; every launch shape (eight,
four and one lane by the number of targets, with and without AV cleaning) has to reproduce them."""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STAGES = {"XMass": ("xm",), "VeDefGradh": ("kx", "gradh", "prho", "c"),
          "IAD": ("c11", "c12", "c13", "c22", "c23", "c33", "divv", "curlv"), "AVswitches": ("alpha",),
          "MomentumEnergy": ("ax", "ay", "az", "du")}
# per side and AV cleaning: the stages' digests in the order of STAGES
RECORDED = {
    (7, False): ("1b5a4f916927", "90e53248f062", "ce47c2f5a5d6", "1b42cfe5af5d", "0d12f576ad1c"),
    (20, False): ("5d6af9d686a5", "36ec4ce35e9d", "e7e85856baf8", "379aecc50d72", "028fe1391889"),
    (36, False): ("d94c5c36978a", "40082c68e855", "7157c729189a", "4390171dba07", "0af69b7af94d"),
    (45, False): ("58fa0823b6e9", "0be82f2aac88", "725147c89855", "d21e96c5b844", "61bc4f0c5f86"),
    (7, True): ("1b5a4f916927", "90e53248f062", "ce47c2f5a5d6", "1b42cfe5af5d", "08ea347eb1a7"),
    (20, True): ("5d6af9d686a5", "36ec4ce35e9d", "e7e85856baf8", "379aecc50d72", "93ae866dacd2"),
    (36, True): ("d94c5c36978a", "40082c68e855", "7157c729189a", "4390171dba07", "704688eb1919"),
    (45, True): ("58fa0823b6e9", "0be82f2aac88", "725147c89855", "d21e96c5b844", "2b9ad4e774bc"),
}


def stirred(side, av_clean):
    """Every input from additions, multiplications, divisions and square roots of counter-based random numbers, the same
    on every host; masses, temperatures and velocities such that all branches of the pair loops occur."""
    from sphexa_b200 import ic as icm
    f = icm.sedov(side)
    i = np.arange(side ** 3, dtype=np.int64)
    r = [icm.uniform01(11, i, k) for k in range(4)] + [icm.uniform01(12, i, k) for k in range(4)]
    x = f["x"]
    f["h"] = (0.95 + 0.1 * r[0]) * (1.44 / side)
    f["m"] = (1.0 + 0.4 * x * x) * (1.0 + 0.3 * r[1]) / side ** 3
    f["temp"] = (0.5 + r[2]) / icm.ideal_gas_cv(f["params"]["mui"], f["params"]["gamma"])
    f["alpha"] = 0.05 + 0.5 * r[3] * r[3]
    for k, v in enumerate(("vx", "vy", "vz")):
        f[v] = 0.3 * (r[4 + k] - 0.5) - x * (0.5 - x * x)
        f[v[1] + "_m1"] = f[v] * 1e-6
    f["params"]["avClean"] = av_clean
    return f


def digests(side, av_clean):
    from sphexa_b200.simulation import Simulation
    sim = Simulation(stirred(side, av_clean), "mixed")
    sim.compute_forces()
    assert sim.get("divv").min() < 0 < sim.get("divv").max()
    return {s: hashlib.sha1(b"".join(sim.get(f).tobytes() for f in names)).hexdigest()[:12]
            for s, names in STAGES.items()}


@pytest.mark.parametrize("av_clean", [False, True])
@pytest.mark.parametrize("side", [7, 20, 36, 45])
def test_forces_keep_their_bits(cuda_device, side, av_clean):
    assert digests(side, av_clean) == dict(zip(STAGES, RECORDED[side, av_clean]))
