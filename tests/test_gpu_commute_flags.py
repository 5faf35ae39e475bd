"""Dense commutation flags straight from the masks, against the definition.

A warp holds 256 columns (1-2 mask words) or 128 (3-4) and sweeps rows; wider masks
and no mask words take the bit matrix.  Rows start at any byte of the matrix, and
nothing outside it is written.
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
    return ((np.bitwise_count(acc) & 1) == 0).astype(np.uint8)


@pytest.mark.parametrize("n", [0, 1, 64, 65, 192, 256, 257])
@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 31), (9, 127), (33, 128), (8, 129), (65, 255), (64, 256), (40, 257),
                                       (3, 5000), (5000, 3), (1300, 700)])
def test_flags(cuda, n, rows, cols):
    import torch

    rng = np.random.default_rng(zlib.crc32(repr(("flags", n, rows, cols)).encode()))
    if n == 0:
        lx = lz = np.zeros((rows, 0), np.uint64)
        rx = rz = np.zeros((cols, 0), np.uint64)
    else:
        _, lx, lz, lc = random_operator(rng, n, rows, 0.3)
        _, rx, rz, rc = random_operator(rng, n, cols, 0.3)
    want = expected(lx, lz, rx, rz)
    dl, dr = G.operator_on_device(lx, lz, np.zeros(rows, np.complex128)), G.operator_on_device(
        rx, rz, np.zeros(cols, np.complex128))
    for offset in (0, 1, 7):
        out = torch.full((rows * cols + 16,), 9, dtype=torch.uint8, device="cuda")
        capi.call("wg_commutation_flags", 0, (n + 63) // 64, G.ptr(dl[0]), G.ptr(dl[1]), rows, G.ptr(dr[0]),
                  G.ptr(dr[1]), cols, out.data_ptr() + offset, None)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert np.array_equal(got[offset : offset + rows * cols].reshape(rows, cols), want)
        assert (got[:offset] == 9).all() and (got[offset + rows * cols :] == 9).all()
