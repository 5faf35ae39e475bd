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
