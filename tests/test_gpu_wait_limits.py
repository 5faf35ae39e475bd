"""Waits of a kernel for earlier blocks of its own launch: the radix passes' look-back.

A wait that gives up (made short by wg_set_wait_limit) ends the call with
WG_ERR_TIMEOUT and nothing else: what the pass left behind is not used, the device
stays usable and the next call with the default limit gives the oracle's bits.
"""

from __future__ import annotations

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
