"""Device memory that calls take beside their operands and results: what fits in the device
has to go on fitting."""

from __future__ import annotations

import ctypes
import gc

import numpy as np
import pytest

from tests import gpu_util as G
from wolfgang_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture
def peak(cuda):
    """peak(call): the most pool memory in use during the call beyond what was in use before."""
    runtime = pytest.importorskip("cuda.bindings.runtime")
    driver = pytest.importorskip("cuda.bindings.driver")
    attr = runtime.cudaMemPoolAttr
    cuda.zeros(1, device="cuda")
    pool = runtime.cudaDeviceGetDefaultMemPool(0)[1]

    def measure(call):
        gc.collect()
        cuda.cuda.synchronize()
        before = int(runtime.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemCurrent)[1])
        runtime.cudaMemPoolSetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh, driver.cuuint64_t(0))
        call()
        return int(runtime.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh)[1]) - before

    return measure


def strings(rng, n, T):
    """T strings of few distinct ones: the tables of distinct keys are small beside the sort."""
    w = (n + 63) // 64
    pool = rng.integers(0, 1 << 63, size=(2, 40, w), dtype=np.uint64)
    pool[:, :, -1] &= np.uint64((1 << (n - 64 * (w - 1))) - 1)
    return pool[0][rng.integers(0, 40, size=T)], pool[1][rng.integers(0, 40, size=T)]


@pytest.mark.parametrize("n", [60, 100, 150])
def test_batch_create(cuda, peak, n):
    """Keys twice (16 K bytes a product for K = 1 + 2 W words) and four 32-bit numbers."""
    from wolfgang_b200.products import ProductsBatch

    rng = np.random.default_rng(n)
    T, K = 2000, 1 + 2 * ((n + 63) // 64)
    pairs = [tuple((n, *strings(rng, n, T), rng.normal(size=T) + 0j) for _ in range(2)) for _ in range(2)]
    kept = []
    used = peak(lambda: kept.append(ProductsBatch(pairs)))
    assert used < (16 * K + 16) * 2 * T * T
    kept[0].close()


@pytest.mark.parametrize("n", [60, 120, 190, 250])
def test_grouping_order(cuda, peak, n):
    rng = np.random.default_rng(n)
    T, w = 400_000, (n + 63) // 64
    x, z = strings(rng, n, T)
    dx, dz, _ = G.operator_on_device(x, z, np.zeros(T, np.complex128))
    order, sizes, count = np.empty(T, np.uint64), np.zeros(T, np.uint64), ctypes.c_size_t(0)
    to = ctypes.POINTER(ctypes.c_size_t)
    used = peak(lambda: capi.call("wg_group_commuting", 0, w, T, G.ptr(dx), G.ptr(dz), 0, order.ctypes.data_as(to),
                                  sizes.ctypes.data_as(to), ctypes.byref(count), None))
    assert used < (16 * (1 + 2 * w) + 16) * T


@pytest.mark.parametrize("n,T", [(20, 1_400_000), (100, 900_000)])
def test_simplify(cuda, peak, n, T):
    """A code, a sum and two item numbers a term, and the packed key (8 bytes for 64 of the 2 n
    varying bits); the sizes keep the call below the 64 MiB from which the workspace, which
    stays for later calls, takes its place."""
    bytes_a_term = 32 + 8 * ((2 * n + 63) // 64)
    rng = np.random.default_rng(n)
    x, z = strings(rng, n, T)
    dx, dz, dc = G.operator_on_device(x, z, rng.normal(size=T) + 0j)
    out = [ctypes.c_void_p() for _ in range(3)]
    terms = ctypes.c_size_t()
    used = peak(lambda: capi.call("wg_simplify", 0, (n + 63) // 64, T, G.ptr(dx), G.ptr(dz), G.ptr(dc), 1e-12, 0.0,
                                  *(ctypes.byref(p) for p in out), ctypes.byref(terms), None))
    assert 0 < terms.value <= 1600 and used < (bytes_a_term + 3) * T
    for p in out:
        capi.call("wg_free", 0, p, None)


@pytest.mark.parametrize("n", [20, 100])
def test_products(cuda, peak, n):
    rng = np.random.default_rng(n)
    T = 1300
    x, z = strings(rng, n, T)
    dx, dz, dc = G.operator_on_device(x, z, rng.normal(size=T) + 0j)
    side = G.ptr(dx), G.ptr(dz), G.ptr(dc), T
    out = [ctypes.c_void_p() for _ in range(3)]
    terms = ctypes.c_size_t()
    used = peak(lambda: capi.call("wg_pauli_products", 0, (n + 63) // 64, *side, *side, capi.WG_PRODUCTS_SIMPLIFY,
                                  1e-12, 0.0, *(ctypes.byref(p) for p in out), ctypes.byref(terms), None))
    assert terms.value > 0 and used < (32 + 3) * T * T + 48 * terms.value
    for p in out:
        capi.call("wg_free", 0, p, None)


_GIVE_BACK = """
import ctypes, numpy as np, torch
from wolfgang_b200 import capi
n, T = 20, 20_000_000
x = torch.randint(0, 1 << n, (T, 1), device="cuda") & 1023
z = torch.zeros_like(x)
c = torch.zeros(T, dtype=torch.complex128, device="cuda") + 1
out, terms = [ctypes.c_void_p() for _ in range(3)], ctypes.c_size_t()
def simplify():
    torch.cuda.synchronize()
    capi.call("wg_simplify", 0, 1, T, x.data_ptr(), z.data_ptr(), c.data_ptr(), 1e-12, 0.0,
              *(ctypes.byref(p) for p in out), ctypes.byref(terms), None)
    assert terms.value == 1024
    for p in out:
        capi.call("wg_free", 0, p, None)
simplify()
torch.cuda.empty_cache()
filler = torch.empty(torch.cuda.mem_get_info()[0] - (2 << 30), dtype=torch.uint8, device="cuda")
free = torch.cuda.mem_get_info()[0]
held = 40 * T  # the workspace of the call above, at least
p = ctypes.c_void_p()
capi.call("wg_malloc", 0, free + held // 2, None, ctypes.byref(p))
capi.call("wg_free", 0, p, None)
simplify()
print("given back")
"""


def test_workspace_is_given_back_when_room_is_short(cuda):
    """With all but 2 GiB of the device taken, an allocation that fits only where the workspace
    of an earlier call lay; the next large call takes a new one."""
    import subprocess
    import sys
    from pathlib import Path

    root = Path(__file__).resolve().parents[1]
    run = subprocess.run([sys.executable, "-c", _GIVE_BACK], cwd=root, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "given back" in run.stdout, run.stderr[-2000:]


@pytest.mark.parametrize("n", [1100, 2000])
def test_small_results_keep_little(cuda, peak, n):
    """100 sums of 8,000 terms that collect to 30 strings or fewer: at most 64 KiB each (blocks
    of masks for all terms would be 2 MB and more, from the pool that is looked at)."""
    runtime = pytest.importorskip("cuda.bindings.runtime")
    rng = np.random.default_rng(n)
    T, w = 8000, (n + 63) // 64
    x, z = strings(rng, n, T)
    x[:], z[:] = x[rng.integers(0, 30, size=T)], z[0]
    dx, dz, dc = G.operator_on_device(x, z, rng.normal(size=T) + 0j)
    results = []

    def used():
        pool = runtime.cudaDeviceGetDefaultMemPool(0)[1]
        return int(runtime.cudaMemPoolGetAttribute(pool, runtime.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)[1])

    cuda.cuda.synchronize()
    before = used()
    for _ in range(100):
        out, terms = [ctypes.c_void_p() for _ in range(3)], ctypes.c_size_t()
        capi.call("wg_simplify", 0, w, T, G.ptr(dx), G.ptr(dz), G.ptr(dc), 1e-12, 0.0, *(ctypes.byref(p) for p in out),
                  ctypes.byref(terms), None)
        assert 0 < terms.value <= 30
        results += out
    assert used() - before < 100 * 65536
    for p in results:
        capi.call("wg_free", 0, p, None)


def test_calls_of_one_size_take_one_time(cuda):
    """Products with the result before still alive, 40 times: small scratch is not cut from the
    blocks that the last results left, so none but the first few calls maps memory (a call of
    1.4 ms took 2 to 5 ms then, three times in four)."""
    import time

    rng = np.random.default_rng(5)
    T = 4096
    x, z = (rng.integers(0, 1 << 20, size=(T, 1), dtype=np.uint64) for _ in range(2))
    dx, dz, dc = G.operator_on_device(x & z, z & np.roll(x, 1), rng.normal(size=T) + 0j)
    side = G.ptr(dx), G.ptr(dz), G.ptr(dc), T
    before, times = [], []
    for i in range(40):
        if i % 13 == 0:  # now and then nothing is alive
            for p in before:
                capi.call("wg_free", 0, p, None)
            before = []
        out, terms = [ctypes.c_void_p() for _ in range(3)], ctypes.c_size_t()
        cuda.cuda.synchronize()
        t = time.perf_counter()
        capi.call("wg_pauli_products", 0, 1, *side, *side, capi.WG_PRODUCTS_SIMPLIFY, 1e-12, 0.0,
                  *(ctypes.byref(p) for p in out), ctypes.byref(terms), None)
        cuda.cuda.synchronize()
        times.append(time.perf_counter() - t)
        for p in before:
            capi.call("wg_free", 0, p, None)
        before = out
    for p in before:
        capi.call("wg_free", 0, p, None)
    late = sorted(times[6:])
    assert sum(t > 1.5 * late[0] for t in late) <= 3
