"""Product batches in which sums are culled: the tiles that meet one keep their sums for
the second writing of the pair."""

from __future__ import annotations

import zlib

import numpy as np
import pytest

from tests.conftest import random_operator
from wolfgang_b200 import capi

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    return a.shape == b.shape and a.tobytes() == b.tobytes()


def check(batch, oracle, n, pairs, rtol=0.0, mode="simplify"):
    for _ in range(2):  # the second run meets the first one's buffers
        batch.run()
    for (A, B), got in zip(pairs, batch.results()):
        raw = oracle.matmul(n, A[1:], B[1:], simplify=False)
        for a, b in zip(got, oracle.simplify(n, *raw, 1e-12, 0.0 if mode == "fused" else rtol)):
            assert same_bits(a, b)


@pytest.mark.parametrize("n", [10, 64, 100, 150])
@pytest.mark.parametrize("mode,rtol", [("simplify", 0.0), ("fused", 0.0), ("simplify", 0.05)])
def test_squares(cuda, oracle, n, mode, rtol):
    """H H: the products of anticommuting terms cancel.  Pairs of several tiles, many pairs in
    a tile, pairs without culls and without products between them."""
    from wolfgang_b200.products import ProductsBatch

    rng = np.random.default_rng(zlib.crc32(repr(("squares", n, mode, rtol)).encode()))
    pairs = []
    for T in [1, 2, 3, 130, 1, 5, 45, 0, 31, 32, 33, 200, 2, 2, 7, 90]:
        H = random_operator(rng, n, T, 0.25 if n <= 10 else 0.05)
        pairs.append((H, H))
        pairs.append((H, random_operator(rng, n, 3, 0.2)))
    batch = ProductsBatch(pairs, mode=mode, rtol=rtol)
    check(batch, oracle, n, pairs, rtol, mode)
    batch.close()


@pytest.mark.parametrize("where", ["first", "last", "all"])
def test_culls_in_one_tile_of_many(cuda, oracle, where):
    """One pair of 60 tiles; coefficients that cancel in the first tile's, the last tile's or
    every sum, so that most tiles do not see the cull."""
    from wolfgang_b200.products import ProductsBatch

    n = 40
    rng = np.random.default_rng(zlib.crc32(where.encode()))
    A, B = random_operator(rng, n, 1500, 0.2), random_operator(rng, n, 41, 0.2)
    # every lhs string twice: a product occurs twice, in order of its key
    x, z, c = (np.concatenate([v, v]) for v in A[1:])
    order = np.lexsort((np.arange(len(c)), z[:, 0], x[:, 0]))
    c[len(A[3]):] *= 0.5
    chosen = {"first": order[:4], "last": order[-4:], "all": order}[where]
    c[chosen] = 0.0
    A = (n, x, z, c)
    batch = ProductsBatch([(A, B)])
    check(batch, oracle, n, [(A, B)])
    batch.close()


def test_the_second_writing_forms_no_products(cuda):
    """Of squares nearly every tile meets a culled sum: the repetition reads sums and keys and
    writes, which is at most two thirds of forming all products, sums and keys again."""
    from wolfgang_b200.products import ProductsBatch

    rng = np.random.default_rng(11)
    pairs = []
    for _ in range(8):
        H = random_operator(rng, 64, 2000, 0.05)
        pairs.append((H, H))
    batch = ProductsBatch(pairs)
    batch.run()
    capi.profile_enable(True)
    try:
        capi.profile_report()
        for _ in range(5):
            batch.run()
        cuda.cuda.synchronize()
        report = capi.profile_report()
    finally:
        capi.profile_enable(False)
    assert report["pbatch_redo_kernel"][1] < 0.67 * report["pbatch_pass_kernel"][1]
    batch.close()
