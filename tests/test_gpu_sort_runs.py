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


@pytest.mark.parametrize("n", [1, 2, 511, 513, 8193, 16_384, 16_385])
@pytest.mark.parametrize("kind", ["floats", "few", "equal", "one digit"])
def test_one_block_sort(cuda_device, kind, n):
    """the sort of the groups' time steps, at the edges of a warp's part and of the block's capacity"""
    import ctypes as C
    import torch
    from sphexa_b200 import lib as L
    sort = L.load()["_ZN4sphb18sortShortKeysAsyncEPmPjmP11CUstream_st"]  # internal: no C entry of its own
    sort.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p]
    rng = np.random.default_rng(n)
    if kind == "floats":
        keys = rng.uniform(1e-7, 1e-3, n).astype(np.float32).view(np.uint32).astype(np.uint64)
    else:
        keys = rng.integers(0, {"few": 7, "equal": 1, "one digit": 256}[kind], n, dtype=np.uint64)
        keys = keys << U(16) if kind == "one digit" else keys + U(0xfffffff0)
    dk = torch.from_numpy(keys.view(np.int64)).cuda()
    dv = torch.arange(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    rc = sort(dk.data_ptr(), dv.data_ptr(), n, None)
    torch.cuda.synchronize()
    if n > 16_384:
        assert rc == L.SPHB_ERR_ARG
        return
    assert rc == L.SPHB_OK
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(dv.cpu().numpy(), order.astype(np.int32))


@pytest.mark.parametrize("initial", [True, False])
@pytest.mark.parametrize("n", [6_000, 70_001, 300_007])
@pytest.mark.parametrize("length", [33, 64, 65, 1000, 2047, 2048, 2049, 5000])
@pytest.mark.parametrize("share", ["one", "some", "all"])
def test_runs_that_a_block_sorts(cuda_device, share, length, n, initial):
    """runs of keys that agree in the upper half, on both sides of what a thread, a block and the sample take; equal keys
    among them, whole runs of one key, and a run at either end"""
    import torch
    from sphexa_b200 import lib as L
    lib = L.load()
    rng = np.random.default_rng(n + length)
    keys = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    part = {"one": length, "some": max(length, n // 5), "all": n}[share]
    cell = np.arange(part, dtype=np.uint64) // U(length)
    low = rng.integers(0, 1 << 32, part, dtype=np.uint64)
    low[::7] = low[0]
    low[cell % U(5) == 1] = U(77)
    keys[:part] = (cell * U(0x2545f491) % U(1 << 31) << U(32)) + low
    keys[part // 2:part] |= U(0x7fffffff00000000) if share == "some" else U(0)
    if not initial:
        keys = rng.permutation(keys)
    order = np.argsort(keys, kind="stable")
    dk = torch.from_numpy(keys.view(np.int64)).cuda()
    values = rng.integers(0, 1 << 31, n, dtype=np.int32)
    dv = torch.from_numpy(values).cuda()
    size = lib.sphb_sort_by_key_scratch_bytes(n)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    L.check(lib.sphb_sort_by_key(L.ptr(dk), L.ptr(dv), n, int(initial), L.ptr(scratch), size, None), "sort")
    torch.cuda.synchronize()
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(dv.cpu().numpy(), order if initial else values[order])
