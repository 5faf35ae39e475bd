"""Waits of a kernel for earlier blocks of its own launch: the radix passes' look-back, and
the grouping stages, which wait as long as some stage makes progress.

A wait that gives up (made short by wg_set_wait_limit) ends the call with
WG_ERR_TIMEOUT and nothing else: what the pass left behind is not used, the device
stays usable and the next call with the default limit gives the oracle's bits.
"""

from __future__ import annotations

import ctypes
import threading
import zlib

import numpy as np
import pytest

from tests import gpu_util as G
from tests.conftest import random_operator
from wolfgang_b200 import capi

pytestmark = pytest.mark.gpu


def seeded(*key):
    return np.random.default_rng(zlib.crc32(repr(key).encode()))


def same(a, b):
    return all(np.ascontiguousarray(x).tobytes() == np.ascontiguousarray(y).tobytes() and x.shape == y.shape
               for x, y in zip(a, b))


@pytest.fixture
def limit():
    yield lambda polls: capi.call("wg_set_wait_limit", polls)
    capi.call("wg_set_wait_limit", 0)


def gives_up(call, attempts=40):
    """Whether one of the attempts ends in WG_ERR_TIMEOUT (no other error is let through)."""
    for _ in range(attempts):
        try:
            call()
        except capi.WGError as e:
            assert e.code == capi.WG_ERR_TIMEOUT and "waited too long" in str(e)
            return True
    return False


@pytest.mark.parametrize("n,T", [(20, 3_000_000), (100, 2_000_000)])
def test_look_back_that_gives_up(cuda, oracle, limit, n, T):
    """Keys that are their codes, and codes that may tie (the reduction would read the keys)."""
    _, x, z, c = random_operator(seeded("look-back", n, T), n, T, 0.25 if n <= 20 else 0.1, T // 4)
    want = oracle.simplify(n, x, z, c, 1e-12, 0.0)
    limit(1)
    assert gives_up(lambda: G.simplify(n, x, z, c))
    few = x[:1800], z[:1800], c[:1800]
    assert gives_up(lambda: G.products(n, few, few))
    limit(0)
    assert same(G.simplify(n, x, z, c), want)


def test_limit_is_the_threads_own(cuda, oracle, limit):
    n, T = 20, 600_000
    _, x, z, c = random_operator(seeded("threads"), n, T, 0.25, T // 4)
    want, got = oracle.simplify(n, x, z, c, 1e-12, 0.0), []
    limit(1)
    worker = threading.Thread(target=lambda: got.append(G.simplify(n, x, z, c)))
    worker.start()
    worker.join()
    assert got and same(got[0], want)


def group(n, x, z, mode):
    w, T = (n + 63) // 64, len(x)
    dx, dz, _ = G.operator_on_device(x, z, np.zeros(T, np.complex128))
    order, sizes, count = np.empty(T, np.uint64), np.zeros(T, np.uint64), ctypes.c_size_t(0)
    to = ctypes.POINTER(ctypes.c_size_t)
    capi.call("wg_group_commuting", 0, w, T, G.ptr(dx), G.ptr(dz), 1 if mode == "full" else 0,
              order.ctypes.data_as(to), sizes.ctypes.data_as(to), ctypes.byref(count), None)
    return order, sizes[: count.value]


@pytest.mark.parametrize("mode,T", [("qwc", 400_000), ("full", 20_000)])
def test_a_stage_that_sees_no_term(cuda, limit, mode, T):
    """Z strings all commute: the first stage of 32 groups takes every term, and the second
    waits for as long as that takes -- about 16 ms and more, many times the limit of 2,000
    polls (of 64 ns and a read), during which the first takes batch after batch."""
    n = 40
    rng = seeded("no term", mode)
    z = rng.integers(0, 1 << n, size=(T, 1), dtype=np.uint64)
    x = np.zeros_like(z)
    weight = np.array([int(v).bit_count() for v in z[:, 0]])
    limit(2000)
    order, sizes = group(n, x, z, mode)
    assert sizes.tolist() == [T]
    assert np.array_equal(order, np.lexsort((np.arange(T), z[:, 0], -weight)).astype(np.uint64))
