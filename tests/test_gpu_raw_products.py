"""Products that are not collected, at every kind of width: 0, 1, 2 and more mask words."""

from __future__ import annotations

import zlib

import numpy as np
import pytest

from tests import gpu_util as G
from tests.conftest import random_operator
from wolfgang_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 5, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("nl,nr", [(1, 1), (1, 700), (513, 1), (37, 41), (300, 1001)])
def test_raw_products(cuda, oracle, n, nl, nr):
    rng = np.random.default_rng(zlib.crc32(repr(("raw", n, nl, nr)).encode()))
    A, B = random_operator(rng, n, nl, 0.2), random_operator(rng, n, nr, 0.2)
    want = oracle.matmul(n, A[1:], B[1:], simplify=False)
    for got, ref in zip(G.products(n, A[1:], B[1:], capi.WG_PRODUCTS_RAW), want):
        assert np.ascontiguousarray(got).tobytes() == np.ascontiguousarray(ref).tobytes()
