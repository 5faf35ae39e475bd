"""The commutation bit matrix from the columns' planes, against the definition.

A CTA takes equal runs of (block of 2,048 or 4,096 columns, row) pairs; rows of up to
12 set qubits are listed beforehand, longer ones word by word; outputs of a pitch that
does not divide by a lane's words are written word by word.  Nothing beyond a row's
words is written.
"""

from __future__ import annotations

import zlib

import numpy as np
import pytest

from tests import gpu_util as G
from tests.conftest import random_operator
from wolfgang_b200 import capi

pytestmark = pytest.mark.gpu


def expected(lx, lz, rx, rz):
    acc = np.zeros((len(lx), len(rx)), np.uint64)
    for w in range(lx.shape[1]):
        acc ^= (lx[:, w, None] & rz[None, :, w]) ^ (lz[:, w, None] & rx[None, :, w])
    return (np.bitwise_count(acc) & 1) == 0


@pytest.fixture
def tuner(cuda):
    mode = capi.autotune_mode()
    capi.autotune_clear()
    capi.autotune_mode(capi.WG_TUNE_CACHED)
    yield capi
    capi.autotune_clear()
    capi.autotune_mode(mode)


@pytest.mark.parametrize("n,p", [(20, 0.3), (64, 0.02), (64, 0.9), (128, 0.05), (128, 0.4), (190, 0.02), (256, 0.03),
                                 (256, 0.6)])
@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 33), (65, 2048), (64, 2049), (700, 4096), (33, 4127), (2500, 8200)])
def test_planes(tuner, n, p, rows, cols):
    rng = np.random.default_rng(zlib.crc32(repr(("planes", n, p, rows, cols)).encode()))
    _, lx, lz, _ = random_operator(rng, n, rows, p)
    _, rx, rz, _ = random_operator(rng, n, cols, p)
    want = expected(lx, lz, rx, rz)
    w, words = (n + 63) // 64, (cols + 31) // 32
    lg = lambda k: (k - 1).bit_length()  # noqa: E731
    left, right = (lx, lz), (rx, rz)
    for candidate in range(1, 5):
        tuner.autotune_import(f"commute {w} {lg(rows)} {lg(cols)} {candidate}\n")
        for pitch in (words, words + 1, (words + 3) // 4 * 4):
            got = G.commutation_bits(n, left, right, algo=0, pitch=pitch)
            assert np.array_equal(G.unpack_bits(got[:, :words].copy(), cols), want)
            tail = np.uint32(0) if cols % 32 == 0 else got[:, words - 1] >> np.uint32(cols % 32)
            assert not np.any(tail)
            assert (got[:, words:] == np.uint32(0xFFFFFFFF)).all()
    assert np.array_equal(G.unpack_bits(G.commutation_bits(n, left, right, algo=2), cols), want)
