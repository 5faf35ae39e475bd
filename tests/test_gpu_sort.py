"""simplify and products around the edges of the sorted path, against the oracle.

One CTA takes up to 8,192 items; above, pairs are sorted in tiles of 4,096 and
reduced in tiles of 1,024 with 256 items staged behind each.  Keys of at most 64
varying bits are sorted by those bits, wider ones by codes that can tie: runs of
equal codes and unequal keys are put in order by a thread (up to 16 items) or by
the whole CTA, and where that is not enough the keys are sorted by all their words.
"""

from __future__ import annotations

import zlib

import numpy as np
import pytest

from tests import gpu_util as G
from tests.conftest import random_operator

pytestmark = pytest.mark.gpu


def seeded(*key):
    return np.random.default_rng(zlib.crc32(repr(key).encode()))


def same(a, b):
    return all(np.ascontiguousarray(x).tobytes() == np.ascontiguousarray(y).tobytes() and x.shape == y.shape
               for x, y in zip(a, b))


def coefficients(rng, T):
    return rng.normal(size=T) + 1j * rng.normal(size=T)


@pytest.mark.parametrize("n,pool", [(20, None), (70, 900), (200, 3000), (300, None)])
@pytest.mark.parametrize("T", [1, 2, 33, 1025, 8191, 8192, 8193, 4096 * 3, 4096 * 3 + 1, 2048 * 9 - 1])
def test_sizes(cuda, oracle, n, pool, T):
    rng = seeded("sizes", n, T)
    _, x, z, c = random_operator(rng, n, T, 0.1, pool)
    assert same(G.simplify(n, x, z, c, 1e-12, 0.0), oracle.simplify(n, x, z, c, 1e-12, 0.0))
    assert same(G.simplify(n, x, z, c, 1e-3, 0.05), oracle.simplify(n, x, z, c, 1e-3, 0.05))


@pytest.mark.parametrize("run", [300, 1024, 1279, 1280, 1281, 2305, 9000])
def test_runs_across_tiles(cuda, oracle, run):
    """Runs of one key that end before, at and behind the staged items."""
    rng = seeded("runs", run)
    n, T = 30, 20000
    x = rng.integers(0, 1 << 30, size=(T, 1), dtype=np.uint64)
    z = np.zeros((T, 1), np.uint64)
    for k, start in enumerate((0, 9500)):
        x[start : start + run] = np.uint64((1 << 29) + 77 * k)
    perm = rng.permutation(T)
    x, z, c = x[perm], z[perm], coefficients(rng, T)
    assert same(G.simplify(n, x, z, c), oracle.simplify(n, x, z, c))


@pytest.mark.parametrize("tails,copies", [(2, 3), (3, 6), (9, 2), (40, 3), (700, 3), (900, 5), (3000, 1)])
@pytest.mark.parametrize("deep", [False, True])
def test_tied_codes(cuda, oracle, tails, copies, deep):
    """Keys that agree in their first 14 (deep: 40) set bits and differ behind:
    runs put in order by a thread, by a CTA, and by all words."""
    rng = seeded("ties", tails, copies, deep)
    n = 256
    lead = 40 if deep else 14
    head = np.zeros((1, 4), np.uint64)
    for q in np.sort(rng.choice(120, size=lead, replace=False)):
        head[0, q // 64] |= np.uint64(1) << np.uint64(q % 64)
    tail = np.zeros((tails, 4), np.uint64)
    tail[:, 3] = rng.permutation(1 << 16)[:tails].astype(np.uint64) << np.uint64(8)
    x = np.repeat(head | tail, copies, axis=0)
    _, ox, oz, _ = random_operator(rng, n, 12000, 0.03)
    x = np.concatenate([x, ox])
    z = np.concatenate([np.zeros((tails * copies, 4), np.uint64), oz])
    T = len(x)
    perm = rng.permutation(T)
    x, z, c = x[perm], z[perm], coefficients(rng, T)
    assert same(G.simplify(n, x, z, c), oracle.simplify(n, x, z, c))


@pytest.mark.parametrize("n,nl,nr", [(6, 1, 8193), (9, 8193, 1), (64, 97, 131), (130, 90, 91), (190, 128, 65), (0, 100, 100)])
def test_products(cuda, oracle, n, nl, nr):
    rng = seeded("products", n, nl, nr)
    A = random_operator(rng, n, nl, 0.06)
    B = random_operator(rng, n, nr, 0.06)
    raw = oracle.matmul(n, A[1:], B[1:], simplify=False)
    assert same(G.products(n, A[1:], B[1:]), oracle.simplify(n, *raw, 1e-12, 0.0))
    assert same(G.products(n, A[1:], B[1:], atol=1e-6, rtol=0.1), oracle.simplify(n, *raw, 1e-6, 0.1))


@pytest.mark.parametrize("T", [700, 9000])
@pytest.mark.parametrize("bad", [np.inf, np.nan, complex(1e308, 1.7e308), complex(np.nan, np.inf)])
def test_not_finite(cuda, oracle, T, bad):
    rng = seeded("bad", T, bad)
    n, x, z, c = random_operator(rng, 40, T, 0.2, T // 5)
    c[T // 3] = bad
    for rtol in (0.0, 0.5):
        assert same(G.simplify(n, x, z, c, 1e-12, rtol), oracle.simplify(n, x, z, c, 1e-12, rtol))


@pytest.mark.parametrize("T", [1, 2, 3, 63, 64, 65, 127, 129, 1024, 1900, 2047, 2048, 2049])
@pytest.mark.parametrize("windows", [(0, 0, 0, 0), (1, 0, 0, 0), (5, 6, 0, 0), (26, 27, 0, 0), (27, 27, 0, 0),
                                     (53, 0, 0, 0), (54, 0, 0, 0), (13, 13, 13, 14), (2, 0, 0, 52)])
def test_windows_of_small_calls(cuda, oracle, T, windows):
    """Up to 2,048 items whose varying bits lie in windows of 53 bits together are sorted as
    one value with their number; constant bits within and beside the windows; duplicates."""
    rng = seeded("windows", T, windows)
    base = rng.integers(0, 1 << 62, size=4, dtype=np.uint64)
    words = np.repeat(base[None, :], T, axis=0)
    for k, width in enumerate(windows):
        if width:
            low = int(rng.integers(0, 63 - width)) if width < 63 else 0
            pool = rng.integers(0, 1 << width, size=max(1, T // 3), dtype=np.uint64)
            pool[0], pool[-1] = 0, (1 << width) - 1
            mask = np.uint64(((1 << width) - 1) << low)
            words[:, k] = (words[:, k] & ~mask) | (rng.choice(pool, size=T) << np.uint64(low))
    order = (0, 2), (1, 3)  # key order x0, z0, x1, z1
    x, z = (np.ascontiguousarray(words[:, list(o)]) for o in order)
    c = coefficients(rng, T)
    n = 126
    assert same(G.simplify(n, x, z, c), oracle.simplify(n, x, z, c))
    if windows[2] == windows[3] == 0:
        assert same(G.simplify(62, x[:, :1], z[:, :1], c), oracle.simplify(62, x[:, :1].copy(), z[:, :1].copy(), c))
