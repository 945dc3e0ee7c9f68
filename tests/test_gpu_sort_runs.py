"""The key sort by the upper digits and a repair of the runs that agree in them, against numpy's stable sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = np.uint64


def _keys(kind, n, rng):
    k = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    if kind == "runs32":  # runs of 32 that agree in the upper half, the longest that one thread sorts
        k = (np.arange(n, dtype=np.uint64) // U(32) << U(33)) + rng.integers(0, 1 << 33, n, dtype=np.uint64) % U(1 << 32)
    if kind == "runs33":
        k = (np.arange(n, dtype=np.uint64) // U(33) << U(33)) + rng.integers(0, 1 << 32, n, dtype=np.uint64)
    if kind == "pairs":
        k = k[rng.integers(0, n, n)] ^ rng.integers(0, 4, n, dtype=np.uint64)
    if kind == "equal halves":  # a long run in order beside spread keys
        k[: n // 2] = U(0x1234567812345678)
    if kind == "dense":  # everything in a few cells of the upper digits: the full sort
        k = (rng.integers(0, 3, n, dtype=np.uint64) << U(60)) + rng.integers(0, 1 << 40, n, dtype=np.uint64) % U(1 << 33)
    if kind == "top bit":
        k[::3] |= U(1 << 63)
    if kind == "few digits":  # trivial digits between the sorted ones
        k &= U(0x7f00ff00ff00ff0f)
    return k if kind.startswith("runs") and n % 2 else rng.permutation(k)


@pytest.mark.parametrize("n", [2, 31, 33, 4097, 100_003])
@pytest.mark.parametrize("kind", ["spread", "runs32", "runs33", "pairs", "equal halves", "dense", "top bit",
                                  "few digits"])
def test_sort_by_key_matches_the_stable_sort(cuda_device, kind, n):
    import torch
    from sphexa_b200 import lib as L
    lib = L.load()
    keys = _keys(kind, n, np.random.default_rng(n))
    order = np.argsort(keys, kind="stable")
    dk = torch.from_numpy(keys.view(np.int64)).cuda()
    values = np.arange(n, dtype=np.int32) * 3
    dv = torch.from_numpy(values).cuda()
    size = lib.sphb_sort_by_key_scratch_bytes(n)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    L.check(lib.sphb_sort_by_key(L.ptr(dk), L.ptr(dv), n, 0, L.ptr(scratch), size, None), "sort")
    torch.cuda.synchronize()
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(dv.cpu().numpy(), values[order])
