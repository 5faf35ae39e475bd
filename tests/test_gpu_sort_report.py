"""wg_last_sort_algorithm tells what ran: the kernels of a call, as the library's own timing
lists them, are those of the sort that it reports."""

from __future__ import annotations

import zlib

import numpy as np
import pytest

from tests import gpu_util as G
from tests.conftest import random_operator
from wolfgang_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture
def algo():
    yield capi.set_sort_algorithm
    capi.set_sort_algorithm(capi.WG_SORT_AUTO)


def run(n, T, setting, algo):
    rng = np.random.default_rng(zlib.crc32(repr((n, T)).encode()))
    _, x, z, c = random_operator(rng, n, T, 0.25 if n <= 32 else 0.05, T // 3)
    algo(setting)
    capi.profile_enable(True)
    try:
        capi.profile_report()
        out = G.simplify(n, x, z, c)
        kernels = set(capi.profile_report())
    finally:
        capi.profile_enable(False)
    return out, kernels, capi.last_sort_algorithm()


@pytest.mark.parametrize("n,T", [(20, 3000), (20, 20_000), (20, 1_100_000), (70, 20_000), (100, 1_100_000), (190, 30_000)])
def test_reported_sort_ran(cuda, algo, n, T):
    got, kernels, told = run(n, T, capi.WG_SORT_AUTO, algo)
    codes = 2 * n > 64 and T > 8192
    assert told == (capi.WG_SORT_BUCKET if codes else capi.WG_SORT_LSD)
    assert "bucket_final_kernel" not in kernels and "word_kernel" not in kernels
    assert ("small_kernel" in kernels) == (T <= 8192) and ("code_kernel" in kernels) == (T > 8192)
    want, kernels, told = run(n, T, capi.WG_SORT_LSD, algo)
    assert told == capi.WG_SORT_LSD
    assert ("word_kernel" in kernels) == codes and ("code_kernel" in kernels) == (T > 8192 and not codes)
    assert all(a.tobytes() == b.tobytes() for a, b in zip(got, want))
