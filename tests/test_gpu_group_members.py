"""Full-mode groups with more members than a stage keeps in shared memory (320 / words):
the others lie in blocks of 128 in device memory."""

from __future__ import annotations

import ctypes
import time
import zlib

import numpy as np
import pytest

from tests import gpu_util as G
from wolfgang_b200 import capi

pytestmark = pytest.mark.gpu


def groups(n, x, z):
    w, T = (n + 63) // 64, len(x)
    dx, dz, _ = G.operator_on_device(x, z, np.zeros(T, np.complex128))
    order, sizes, count = np.empty(T, np.uint64), np.zeros(T, np.uint64), ctypes.c_size_t(0)
    to = ctypes.POINTER(ctypes.c_size_t)
    G.torch().cuda.synchronize()
    t = time.perf_counter()
    capi.call("wg_group_commuting", 0, w, T, G.ptr(dx), G.ptr(dz), 1, order.ctypes.data_as(to),
              sizes.ctypes.data_as(to), ctypes.byref(count), None)
    t = time.perf_counter() - t
    return [v.astype(int).tolist() for v in np.split(order, np.cumsum(sizes[: count.value])[:-1].astype(int))], t


def strings(rng, n, T):
    """T words of n random bits."""
    bits = rng.random((T, n)) < 0.5
    words = np.zeros((T, (n + 63) // 64), np.uint64)
    for q in range(n):
        words[:, q // 64] |= bits[:, q].astype(np.uint64) << np.uint64(q % 64)
    return words


@pytest.mark.parametrize("n", [24, 100, 190, 250])
@pytest.mark.parametrize("beyond", [-1, 0, 1, 31, 32, 33, 127, 128, 129, 255, 257, 700])
def test_block_edges(cuda, oracle, n, beyond):
    """One group of `beyond` more members than fit, all Z, and X strings that meet them."""
    rng = np.random.default_rng(zlib.crc32(repr(("edges", n, beyond)).encode()))
    T = 320 // ((n + 63) // 64) + beyond
    z = strings(rng, n, T)
    x = np.zeros_like(z)
    few = strings(rng, n, 40)
    few[:, :] &= few[rng.integers(0, 40, size=40)]  # lighter: they come last and meet the whole group
    x, z = np.concatenate([x, few]), np.concatenate([z, np.zeros_like(few)])
    perm = rng.permutation(T + 40)
    x, z = np.ascontiguousarray(x[perm]), np.ascontiguousarray(z[perm])
    assert groups(n, x, z)[0] == oracle.group_commuting(n, x, z, "full")


@pytest.mark.parametrize("n,T", [(12, 3000), (70, 2500), (150, 2000), (250, 1500)])
def test_several_long_groups(cuda, oracle, n, T):
    """Z strings, X strings and XZ strings with even overlaps: their groups grow in turns."""
    rng = np.random.default_rng(zlib.crc32(repr(("several", n, T)).encode()))
    kind = rng.integers(0, 3, size=T)
    a, b = strings(rng, n, T), strings(rng, n, T)
    x = np.where((kind > 0)[:, None], a, np.uint64(0))
    z = np.where((kind == 0)[:, None], a, np.where((kind == 1)[:, None], np.uint64(0), a))
    z[kind == 2] ^= b[kind == 2] & np.uint64(3)
    assert groups(n, x, z)[0] == oracle.group_commuting(n, x, z, "full")


def test_long_lists_are_not_followed_link_by_link(cuda):
    """8,192 Z strings on 250 qubits, T^2 / 2 pairs of members: a lane that followed a list
    link by link, 31 terms at once, would take 110 ms at 200 cycles a link.  Half of that
    is the limit (a member per lane needs a thirtieth)."""
    rng = np.random.default_rng(7)
    T = 8192
    z = strings(rng, 250, T)
    x = np.zeros_like(z)
    groups(250, x, z)
    out, best = None, 1e9
    for _ in range(3):
        out, t = groups(250, x, z)
        best = min(best, t)
    assert len(out) == 1 and len(out[0]) == T
    assert best < 0.5 * (T * T / 2) / 31 * 200 / 1.965e9
