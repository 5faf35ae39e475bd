"""Expectation and its adjoint around the edges of the tiles, against the oracle.

Tiles hold 2^12 amplitudes (2^9 to 2^12 for fewer qubits); terms of one x go in
pieces of at most 8; classes of x above the tile share a source tile.  Sums of N
products of numbers below 1 in FP64 are off by at most N 2^-53 times their size:
with norms of 1 and at most 2^15 amplitudes and 2,000 terms of size about 1 that
is below 1e-11, the bound used here.
"""

from __future__ import annotations

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 1e-11


def operator(rng, n, T, patterns):
    """T terms whose x are among `patterns` masks (0 among them), any z."""
    if n == 0:
        return np.zeros((T, 0), np.uint64), np.zeros((T, 0), np.uint64)
    full = (1 << n) - 1
    pool = np.unique(np.concatenate([[0], rng.integers(0, full + 1, size=max(1, patterns - 1))]).astype(np.uint64))
    x = rng.choice(pool, size=T).astype(np.uint64).reshape(T, 1)
    z = rng.integers(0, full + 1, size=(T, 1)).astype(np.uint64)
    return x, z


@pytest.mark.parametrize("real", [True, False])
@pytest.mark.parametrize("n,T,patterns", [(0, 3, 1), (1, 5, 2), (4, 40, 5), (8, 300, 3), (9, 700, 20), (10, 60, 60),
                                          (11, 100, 7), (12, 300, 9), (12, 1, 1), (13, 400, 12), (14, 120, 50), (15, 33, 2)])
def test_tiles(cuda, oracle, n, T, patterns, real):
    torch = cuda
    from wolfgang_b200.expectation import ExpectationPlan

    rng = np.random.default_rng(zlib.crc32(repr(("tiles", n, T, patterns)).encode()))
    x, z = operator(rng, n, T, patterns)
    c = (rng.normal(size=T) + (0.0 if real else 1j * rng.normal(size=T))).astype(np.complex128) / np.sqrt(T)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    plan = ExpectationPlan((n, x, z, c))
    res, ev, hp = plan.run(torch.from_numpy(psi).cuda(), terms=True, hpsi=True)
    assert abs(complex(*res.tolist()) - oracle.expectation(n, x, z, c, psi)) <= BOUND
    assert np.max(np.abs(ev.cpu().numpy() - oracle.term_expectations(n, x, z, psi))) <= BOUND
    assert np.max(np.abs(hp.cpu().numpy() - oracle.hpsi(n, x, z, c, psi))) <= BOUND
    # complex64 storage at an address that is a multiple of 8 only, against the same stored amplitudes
    room = torch.zeros((1 << n) + 1, dtype=torch.complex64, device="cuda")
    room[1:] = torch.from_numpy(psi.astype(np.complex64)).cuda()
    wide = psi.astype(np.complex64).astype(np.complex128)
    res, ev, hp = plan.run(room[1:], terms=True, hpsi=True)
    assert np.max(np.abs(ev.cpu().numpy() - oracle.term_expectations(n, x, z, wide))) <= BOUND
    assert np.max(np.abs(hp.cpu().numpy() - oracle.hpsi(n, x, z, c, wide))) <= BOUND
    # new coefficients, from real to complex or back
    c2 = (rng.normal(size=T) + (1j * rng.normal(size=T) if real else 0.0)).astype(np.complex128) / np.sqrt(T)
    plan.set_coefficients(torch.from_numpy(c2).cuda())
    res, _, hp = plan.run(torch.from_numpy(psi).cuda(), hpsi=True)
    assert abs(complex(*res.tolist()) - oracle.expectation(n, x, z, c2, psi)) <= BOUND
    assert np.max(np.abs(hp.cpu().numpy() - oracle.hpsi(n, x, z, c2, psi))) <= BOUND
    plan.close()


@pytest.mark.parametrize("n,T,patterns", [(3, 1, 1), (12, 512, 60), (12, 513, 60), (13, 1, 1), (13, 3, 3), (14, 40, 40),
                                          (15, 16, 16), (16, 12, 6), (16, 700, 300)])
def test_few_terms_a_class_and_single_calls(cuda, oracle, n, T, patterns):
    """Chunks whose pieces read the paired tile themselves; sums joined in one block up to
    512 terms; one pair in the kernel's parameter or several in a table, with and without
    outputs: the same bits."""
    torch = cuda
    from wolfgang_b200.expectation import ExpectationBatch, ExpectationPlan

    rng = np.random.default_rng(zlib.crc32(repr(("calls", n, T, patterns)).encode()))
    x, z = operator(rng, n, T, patterns)
    c = rng.normal(size=T) / np.sqrt(T)
    host = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    host /= np.linalg.norm(host)
    other = ExpectationPlan((4, x[:3] & np.uint64(15), z[:3] & np.uint64(15), c[:3].astype(np.complex128)))
    for dtype in (np.complex128, np.complex64):
        stored = host.astype(dtype)
        psi, wide = torch.from_numpy(stored).cuda(), stored.astype(np.complex128)
        plan = ExpectationPlan((n, x, z, np.zeros(T, np.complex128)))
        plan.set_coefficients(torch.from_numpy(c).cuda())  # real ones as they are
        res, ev, hp = plan.run(psi, terms=True, hpsi=True)
        assert abs(complex(*res.tolist()) - oracle.expectation(n, x, z, c.astype(np.complex128), wide)) <= BOUND
        assert np.max(np.abs(ev.cpu().numpy() - oracle.term_expectations(n, x, z, wide))) <= BOUND
        assert np.max(np.abs(hp.cpu().numpy() - oracle.hpsi(n, x, z, c.astype(np.complex128), wide))) <= BOUND
        assert plan.run(psi)[0].tolist() == res.tolist()
        small = torch.from_numpy(stored[:16].copy()).cuda()
        batch = ExpectationBatch([other, plan], [small, psi])
        batch.run()
        assert batch.values[1].tolist() == res.tolist()
        assert torch.equal(batch.term_values[1][:T], ev) and torch.equal(batch.hpsi[1], hp)
        one = ExpectationBatch([plan], [psi])
        one.run()
        assert one.values[0].tolist() == res.tolist() and torch.equal(one.hpsi[0], hp)
        plan.set_coefficients(torch.from_numpy(c.astype(np.complex128)).cuda())
        again = plan.run(psi, terms=True, hpsi=True)
        assert again[0].tolist() == res.tolist() and torch.equal(again[2], hp)
        for o in (batch, one, plan):
            o.close()
    other.close()
