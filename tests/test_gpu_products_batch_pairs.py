"""Product batches of very many small pairs: a position's pair is searched, not walked to."""

from __future__ import annotations

import time
import zlib

import numpy as np
import pytest

from tests.conftest import random_operator

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    return a.shape == b.shape and a.tobytes() == b.tobytes()


def batch_and_operands(n, count, most, **kw):
    from wolfgang_b200.products import ProductsBatch

    rng = np.random.default_rng(zlib.crc32(repr(("pairs", n, count, most)).encode()))
    _, x, z, c = random_operator(rng, n, 4 * most, 0.3, most)
    pairs = []
    for _ in range(count):
        side = []
        for _ in range(2):
            T, at = int(rng.integers(0, most + 1)), int(rng.integers(0, 3 * most))
            side.append((n, x[at : at + T], z[at : at + T], c[at : at + T]))
        pairs.append(tuple(side))
    return ProductsBatch(pairs, **kw), pairs


@pytest.mark.parametrize("n,count,most", [(6, 2500, 1), (12, 1500, 3), (70, 700, 8), (130, 300, 40)])
@pytest.mark.parametrize("rtol", [0.0, 0.2])
def test_small_pairs(cuda, oracle, n, count, most, rtol):
    """Sizes from 0 on, so that pairs without products lie between the others."""
    batch, pairs = batch_and_operands(n, count, most, rtol=rtol)
    batch.run()
    counts = batch.counts()
    step = 1 if most > 3 else 7
    for p in range(0, count, step):
        A, B = pairs[p]
        raw = oracle.matmul(n, A[1:], B[1:], simplify=False)
        want = oracle.simplify(n, *raw, 1e-12, rtol)
        for a, b in zip(batch.result(p, int(counts[p])), want):
            assert same_bits(a, b)
    batch.close()


def test_largest_products_of_many_pairs(cuda):
    """rtol > 0 adds a pass that forms every product and finds its pair by a search of
    15 steps: a few times the run without it, where a walk from the first pair on takes
    thousands of steps a product."""
    times = {}
    for rtol in (0.0, 1e-3):
        batch, _ = batch_and_operands(20, 20000, 3, rtol=rtol)
        best = 1e9
        for _ in range(5):
            cuda.cuda.synchronize()
            t = time.perf_counter()
            batch.run()
            cuda.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        times[rtol] = best
        batch.close()
    assert times[1e-3] < 6 * times[0.0]
