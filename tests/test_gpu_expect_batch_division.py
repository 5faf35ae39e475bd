"""How a batch divides the work of its pairs: chunks of a pair taken together in one forward
item, the splits of a tile one after another in one adjoint item.  Neither may change a bit
of what a plan gives alone, and a batch of many pairs keeps no partial H psi for each."""

from __future__ import annotations

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operator(rng, n, T, patterns):
    full = (1 << n) - 1
    pool = np.unique(np.concatenate([[0], rng.integers(0, full + 1, size=patterns)]).astype(np.uint64))
    return (rng.choice(pool, size=T).astype(np.uint64).reshape(T, 1),
            rng.integers(0, full + 1, size=(T, 1)).astype(np.uint64))


def pairs_of(torch, seed, sizes, dtype):
    from wolfgang_b200.expectation import ExpectationPlan

    rng = np.random.default_rng(zlib.crc32(repr(seed).encode()))
    plans, psis = [], []
    for n, T, patterns in sizes:
        x, z = operator(rng, n, T, patterns)
        c = rng.normal(size=T) + (1j * rng.normal(size=T) if T % 3 == 0 else 0.0)
        plans.append(ExpectationPlan((n, x, z, c.astype(np.complex128))))
        psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        psis.append(torch.from_numpy((psi / np.linalg.norm(psi)).astype(dtype)).cuda())
    return plans, psis


EQUAL = [(n, T, patterns) for n, T, patterns in ((5, 90, 20), (9, 300, 80), (10, 200, 200), (11, 500, 60),
                                                   (12, 300, 150), (13, 260, 260), (14, 90, 12), (15, 60, 60))]


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("sizes", [[e] * 40 for e in EQUAL] + [EQUAL * 5, [EQUAL[2]] * 60 + [(16, 900, 300)],
                                                                [(15, 2000, 400)] + [(12, 1, 1), (13, 16, 16)] * 30,
                                                                [(14, 700, 700)] * 2], ids=lambda s: f"{len(s)}-{'-'.join(map(str, s[0]))}")
def test_same_bits_as_alone(cuda, dtype, sizes):
    torch = cuda
    from wolfgang_b200.expectation import ExpectationBatch

    plans, psis = pairs_of(torch, ("division", sizes), sizes, dtype)
    alone = [p.run(psi, terms=True, hpsi=True) for p, psi in zip(plans, psis)]
    for gradients in (True, False):
        batch = ExpectationBatch(plans, psis, gradients=gradients)
        for _ in range(2):
            batch.run()
        for i, (res, ev, hp) in enumerate(alone):
            assert torch.equal(batch.values[i], res)
            assert torch.equal(batch.term_values[i][: plans[i].T], ev)
            if gradients:
                assert torch.equal(batch.hpsi[i], hp)
        batch.close()
    for p in plans:
        p.close()


def test_many_pairs_keep_no_partial_sums(cuda):
    """256 pairs of 12 qubits: 64 splits each would be 1 GiB of partial H psi."""
    torch = cuda
    runtime = pytest.importorskip("cuda.bindings.runtime")
    from wolfgang_b200.expectation import ExpectationBatch

    plans, psis = pairs_of(torch, "memory", [(12, 400, 200)] * 256, np.complex128)
    torch.cuda.synchronize()
    pool = runtime.cudaDeviceGetDefaultMemPool(0)[1]

    def used():
        return int(runtime.cudaMemPoolGetAttribute(pool, runtime.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)[1])

    before = used()
    batch = ExpectationBatch(plans, psis)
    assert used() - before < 64 << 20
    batch.close()
    for p in plans:
        p.close()
