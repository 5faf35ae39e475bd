"""group_commuting as a pipeline of stages of 32 groups, against the oracle.

Terms reach a stage in batches of 256 (qubit-wise) or 31 (full) and are placed 32
at a time; a full-mode stage keeps 320 / words members of a group in shared memory
and links the others; where the stages that the device holds at once are not
enough, the rest of the terms go through as many again.
"""

from __future__ import annotations

import ctypes
import zlib

import numpy as np
import pytest

from tests import gpu_util as G
from tests.conftest import random_operator
from wolfgang_b200 import capi

pytestmark = pytest.mark.gpu


def groups(n, x, z, mode):
    w, T = (n + 63) // 64, len(x)
    dx, dz, _ = G.operator_on_device(x, z, np.zeros(T, np.complex128))
    order, sizes, count = (ctypes.c_size_t * T)(), (ctypes.c_size_t * T)(), ctypes.c_size_t(0)
    capi.call("wg_group_commuting", 0, w, T, G.ptr(dx), G.ptr(dz), 1 if mode == "full" else 0, order, sizes,
              ctypes.byref(count), None)
    out, at = [], 0
    for k in range(count.value):
        out.append(list(order[at : at + sizes[k]]))
        at += sizes[k]
    return out


@pytest.mark.parametrize("mode", ["qwc", "full"])
@pytest.mark.parametrize("n", [5, 64, 100, 190, 256])
@pytest.mark.parametrize("T", [1, 31, 32, 33, 255, 256, 257, 1100])
def test_batch_edges(cuda, oracle, mode, n, T):
    rng = np.random.default_rng(zlib.crc32(repr(("batches", mode, n, T)).encode()))
    _, x, z, _ = random_operator(rng, n, T, 0.1 if n > 64 else 0.3)
    assert groups(n, x, z, mode) == oracle.group_commuting(n, x, z, mode)


@pytest.mark.parametrize("n,T", [(12, 1000), (256, 700)])
def test_long_member_lists(cuda, oracle, n, T):
    """Z strings all commute; a few others split them late."""
    rng = np.random.default_rng(zlib.crc32(repr(("members", n, T)).encode()))
    _, x, z, _ = random_operator(rng, n, T, 0.3)
    x[: T - 40] = 0
    assert groups(n, x, z, "full") == oracle.group_commuting(n, x, z, "full")


def test_more_groups_than_resident_stages(cuda, oracle):
    rng = np.random.default_rng(zlib.crc32(b"many groups"))
    _, x, z, _ = random_operator(rng, 64, 10500, 0.9)
    want = oracle.group_commuting(64, x, z, "qwc")
    assert len(want) > 2 * 148 * 32
    assert groups(64, x, z, "qwc") == want
