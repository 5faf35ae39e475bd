"""The work that a user of this library has it do, as cases that can be timed.

A case is a dict of plain values; ``kind`` names the public call it goes through:

  gradient   ``expectation.expectation`` and its backward pass: one step of a variational loop
  expect     ``DevicePauliSum.expectation_statevector`` of a state on the GPU
  batch      ``ExpectationBatch.replay``: many uneven (H, psi) pairs from one CUDA graph
  matmul     ``DevicePauliSum.matmul``: all products, equal strings collected
  simplify   ``DevicePauliSum.simplify`` of an operator with repeated strings
  flags      ``DevicePauliSum.commutes_with_device``: one byte per pair
  bits       ``DevicePauliSum.commutes_with_bits``: one bit per pair
  group      ``wg_group_commuting`` of the C interface
  products   ``ProductsBatch.replay``: many uneven products from one CUDA graph

Operators come in three families: "dense" (every qubit non-identity with probability ``p``, as in
the 20-qubit and 128-qubit workloads), "local" (weight uniform in 1..``weight``, as in the products
and batch workloads) and "pattern" (X parts from a few distinct patterns, as in the 26-qubit workload).
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from wolfgang_b200 import PauliSum, capi
from wolfgang_b200.expectation import ExpectationBatch, ExpectationPlan, expectation
from wolfgang_b200.products import ProductsBatch


def listed():
    return [
        # one step of a small variational loop: launches and host work count
        dict(name="gradient 12 qubits", kind="gradient", qubits=12, terms=512, single=False),
        # the differentiable expectation of a large Hamiltonian: both directions, X parts repeat
        dict(name="gradient 24 qubits", kind="gradient", qubits=24, terms=20000, single=False),
        # the value alone, for a dense operator whose X parts hardly repeat
        dict(name="expect 20 qubits", kind="expect", qubits=20, terms=4096, p=0.25, single=False),
        # many small Hamiltonians of uneven size with complex64 states
        dict(name="batch 8-18 qubits", kind="batch", pairs=30, low=8, high=18, most=5000, single=True),
        # a product of two short operators, as in symbolic algebra
        dict(name="matmul 48x40", kind="matmul", qubits=16, lhs=48, rhs=40, family="local", p=0.0, weight=4),
        # H @ H on few qubits: most strings occur more than once
        dict(name="matmul 4096x4096 dense", kind="matmul", qubits=20, lhs=4096, rhs=4096, family="dense", p=0.25, weight=0),
        # a product of two local operators on many qubits: most strings occur once
        dict(name="matmul 8192x8192 local", kind="matmul", qubits=100, lhs=8192, rhs=8192, family="local", p=0.0, weight=4),
        # collecting a long sum whose strings repeat about fifty times
        dict(name="simplify 5000000", kind="simplify", qubits=20, terms=5000000, distinct=100000),
        # a conflict graph of ordinary size, one byte per pair
        dict(name="flags 4099x4099", kind="flags", qubits=20, lhs=4099, rhs=4099, p=0.25),
        # a conflict graph of a large operator, one bit per pair
        dict(name="bits 131072x131072", kind="bits", qubits=128, lhs=131072, rhs=131072, p=0.05),
        # measurement groups of a large operator (qubit-wise commuting, the default mode)
        dict(name="group 65536", kind="group", qubits=128, terms=65536, p=0.05, full=False),
        # commutators of many operators with new coefficients in each step
        dict(name="products 64 pairs", kind="products", qubits=64, pairs=64, low=16, high=4096),
    ]


def _log(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["gradient", "expect", "batch", "matmul", "matmul", "simplify", "flags", "bits", "group", "products"])
    single = rng.random() < 0.4
    if kind == "gradient":
        n = rng.randint(8, 24)
        return dict(kind=kind, qubits=n, terms=_log(rng, 64, 20000), single=single)
    if kind == "expect":
        return dict(kind=kind, qubits=rng.randint(6, 22), terms=_log(rng, 16, 4096), p=rng.choice([0.1, 0.25, 0.5]), single=single)
    if kind == "batch":
        low = rng.randint(6, 12)
        return dict(kind=kind, pairs=rng.randint(2, 30), low=low, high=low + rng.randint(0, 6), most=_log(rng, 200, 5000), single=single)
    if kind == "matmul":
        lhs, rhs = _log(rng, 2, 8192), _log(rng, 2, 8192)
        if rng.random() < 0.5:
            return dict(kind=kind, qubits=rng.randint(6, 40), lhs=lhs, rhs=rhs, family="dense", p=0.25, weight=0)
        return dict(kind=kind, qubits=rng.randint(8, 150), lhs=lhs, rhs=rhs, family="local", p=0.0, weight=rng.randint(2, 6))
    if kind == "simplify":
        terms = _log(rng, 100, 5000000)
        return dict(kind=kind, qubits=rng.randint(10, 120), terms=terms, distinct=max(1, int(terms / math.exp(rng.uniform(0.0, 5.0)))))
    if kind == "flags":
        return dict(kind=kind, qubits=rng.randint(4, 200), lhs=_log(rng, 16, 8192), rhs=_log(rng, 16, 8192), p=rng.choice([0.05, 0.25]))
    if kind == "bits":
        return dict(kind=kind, qubits=rng.randint(20, 250), lhs=_log(rng, 1000, 131072), rhs=_log(rng, 1000, 131072), p=rng.choice([0.05, 0.1, 0.25]))
    if kind == "group":
        full = rng.random() < 0.5
        return dict(kind=kind, qubits=rng.randint(16, 200), terms=_log(rng, 100, 16384 if full else 65536), p=rng.choice([0.05, 0.1]), full=full)
    low = _log(rng, 8, 64)
    return dict(kind=kind, qubits=rng.randint(10, 100), pairs=rng.randint(2, 64), low=low, high=_log(rng, 128, 4096))


# ------------------------------------------------------------------ operators

_DEV = "cuda"


def _generator(seed):
    g = torch.Generator(device=_DEV)
    g.manual_seed(int(seed))
    return g


def _pack(bits):
    """(T, n) bool -> (T, W) int64 words, qubit q in bit q % 64 of word q // 64."""
    T, n = bits.shape
    words = []
    for lo in range(0, n, 64):
        part = bits[:, lo : lo + 64]
        words.append((part.to(torch.int64) << torch.arange(part.shape[1], device=bits.device)).sum(1))
    return torch.stack(words, 1)


def _structure(case):
    """The generator of what is part of the case: its number of results depends on nothing else."""
    return _generator(sum(v * (31 ** i) for i, v in enumerate(case[k] for k in sorted(case) if type(case[k]) is int)) % (1 << 40))


def _relabelling(g, n):
    """An order of the qubits and a cyclic renaming of X, Y and Z on each: other strings with the same products."""
    return torch.randperm(n, generator=g, device=_DEV), torch.randint(0, 3, (n,), generator=g, device=_DEV)


def _strings(g, active, relabel=None):
    """X, Y or Z with equal chance where active."""
    kind = torch.randint(0, 3, active.shape, generator=g, device=_DEV)
    if relabel is not None:
        active, kind = active[:, relabel[0]], (kind[:, relabel[0]] + relabel[1]) % 3
    return _pack(active & (kind < 2)), _pack(active & (kind > 0))


def _coefficients(g, T, real=False):
    c = torch.randn(T, 2, generator=g, device=_DEV, dtype=torch.float64)
    if real:
        c[:, 1] = 0.0
    return torch.view_as_complex(c)


def _dense(g, n, T, p, relabel=None):
    return _strings(g, torch.rand(T, n, generator=g, device=_DEV) < p, relabel)


def _local(g, n, T, weight, relabel=None):
    w = torch.randint(1, min(weight, n) + 1, (T, 1), generator=g, device=_DEV)
    rank = torch.rand(T, n, generator=g, device=_DEV).argsort(1).argsort(1)
    return _strings(g, rank < w, relabel)


def _pattern(g, n, T):
    """X parts of weight 0..4 from about T / 10 patterns; the term's weight is 1..8, the rest of it Z."""
    most = min(4, n)
    count = max(4, T // 10)
    a = torch.randint(0, most + 1, (2 * count, 1), generator=g, device=_DEV)
    sup = torch.rand(2 * count, n, generator=g, device=_DEV).argsort(1).argsort(1) < a
    pat = torch.unique(sup, dim=0)
    pat = pat[torch.randperm(pat.shape[0], generator=g, device=_DEV)[:count]]
    wt = pat.sum(1)
    order = torch.sort(wt, stable=True).indices
    pat, wt = pat[order], wt[order]
    w = torch.randint(1, min(8, n) + 1, (T,), generator=g, device=_DEV)
    fit = torch.searchsorted(wt.contiguous(), w, right=True).clamp(min=1)  # patterns no heavier than the term
    pick = (torch.rand(T, generator=g, device=_DEV) * fit).long().clamp(max=pat.shape[0] - 1)
    on = pat[pick]
    score = torch.rand(T, n, generator=g, device=_DEV).masked_fill(on, 2.0)
    extra = score.argsort(1).argsort(1) < (w - wt[pick]).clamp(min=0)[:, None]
    y = torch.rand(T, n, generator=g, device=_DEV) < 0.5
    return _pack(on), _pack((on & y) | (extra & ~on))


def _state(g, n, single):
    psi = torch.view_as_complex(torch.randn(1 << n, 2, generator=g, device=_DEV, dtype=torch.float64))
    psi = psi / torch.linalg.vector_norm(psi)
    return psi.to(torch.complex64) if single else psi


def _device_sum(n, x, z, c):
    return PauliSum.from_packed(n, x.cpu().numpy().view(np.uint64), z.cpu().numpy().view(np.uint64), c.cpu().numpy()).to_device()


def _sizes(case):
    """Uneven sizes of a batch: part of the case, not of its values."""
    return np.random.default_rng(1000003 * case["pairs"] + case["low"])


def _batch_inputs(case, seed):
    g, r = _generator(seed), _sizes(case)
    out = []
    for _ in range(case["pairs"]):
        n = int(r.integers(case["low"], case["high"] + 1))
        T = int(round(math.exp(r.uniform(math.log(100), math.log(case["most"])))))
        x, z = _local(g, n, T, 6)
        out.append((n, x, z, _coefficients(g, T, real=True), _state(g, n, case["single"])))
    return out


def _products_inputs(case, seed):
    g, fixed, r = _generator(seed), _structure(case), _sizes(case)
    n, out = case["qubits"], []
    relabel = _relabelling(g, n)
    for _ in range(case["pairs"]):
        pair = []
        for T in np.round(np.exp(r.uniform(math.log(case["low"]), math.log(case["high"]), size=2))).astype(int):
            pair.append((n, *_local(fixed, n, int(T), 6, relabel), _coefficients(g, int(T))))
        out.append(tuple(pair))
    return out


def _operator(case, g, T, relabel):
    if case["family"] == "dense":
        return _dense(g, case["qubits"], T, case["p"], relabel)
    return _local(g, case["qubits"], T, case["weight"], relabel)


def _simplify_inputs(case, seed):
    g, fixed = _generator(seed), _structure(case)
    x, z = _local(fixed, case["qubits"], case["distinct"], 8, _relabelling(g, case["qubits"]))
    pick = torch.randint(0, case["distinct"], (case["terms"],), generator=fixed, device=_DEV)
    pick = pick[torch.randperm(case["terms"], generator=g, device=_DEV)]
    return x[pick], z[pick], _coefficients(g, case["terms"])


def _matmul_inputs(case, seed):
    g, fixed = _generator(seed), _structure(case)
    relabel = _relabelling(g, case["qubits"])
    return [(*_operator(case, fixed, T, relabel), _coefficients(g, T)) for T in (case["lhs"], case["rhs"])]


def _gradient_inputs(case, seed):
    g = _generator(seed)
    n, T = case["qubits"], case["terms"]
    x, z = _pattern(g, n, T)
    c = torch.randn(T, generator=g, device=_DEV, dtype=torch.float64) / math.sqrt(T)
    return x, z, c, _state(g, n, case["single"])


def _expect_inputs(case, seed):
    g = _generator(seed)
    x, z = _dense(g, case["qubits"], case["terms"], case["p"])
    return x, z, _coefficients(g, case["terms"]), _state(g, case["qubits"], case["single"])


# ------------------------------------------------------------------ a pass


class _Memory:
    """A view of device memory that keeps its owner alive."""

    def __init__(self, owner, pointer, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(pointer, False), version=2)


def _tensor(owner, pointer, shape, typestr):
    if 0 in shape:
        return torch.empty(shape, dtype={"<i8": torch.int64, "<i4": torch.int32, "<c16": torch.complex128}[typestr], device=_DEV)
    return torch.as_tensor(_Memory(owner, pointer, shape, typestr), device=_DEV)


def _terms(op):
    """The words and coefficients of an operator on the device, where they lie."""
    x, z, c = op._pointers
    T, W = op.num_terms, (op.num_qubits + 63) // 64
    return {"x": _tensor(op, x, (T, W), "<i8"), "z": _tensor(op, z, (T, W), "<i8"), "c": _tensor(op, c, (T,), "<c16")}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "gradient":
        x, z, c, psi = _gradient_inputs(case, seed)
        s.update(plan=ExpectationPlan((case["qubits"], x, z, c.to(torch.complex128))), coeffs=c.requires_grad_(), psi=psi.requires_grad_())
    elif kind == "expect":
        x, z, c, psi = _expect_inputs(case, seed)
        s.update(op=_device_sum(case["qubits"], x, z, c), psi=psi)
    elif kind == "batch":
        pairs = _batch_inputs(case, seed)
        plans = [ExpectationPlan(p[:4]) for p in pairs]
        s.update(batch=ExpectationBatch(plans, [p[4] for p in pairs]))
        s["batch"].capture()
    elif kind == "matmul":
        (lx, lz, lc), (rx, rz, rc) = _matmul_inputs(case, seed)
        s.update(lhs=_device_sum(case["qubits"], lx, lz, lc), rhs=_device_sum(case["qubits"], rx, rz, rc))
    elif kind == "simplify":
        s.update(op=_device_sum(case["qubits"], *_simplify_inputs(case, seed)))
    elif kind in ("flags", "bits"):
        g = _generator(seed)
        for side in ("lhs", "rhs"):
            x, z = _dense(g, case["qubits"], case[side], case["p"])
            s[side] = _device_sum(case["qubits"], x, z, _coefficients(g, case[side]))
    elif kind == "group":
        s["x"], s["z"] = (v.contiguous() for v in _dense(_generator(seed), case["qubits"], case["terms"], case["p"]))
    else:
        batch = ProductsBatch(_products_inputs(case, seed))
        batch.capture()
        # the result slots of all pairs lie one after another
        x, z, c, cap = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_size_t()
        capi.call("wg_products_batch_result", batch.handle, 0, ctypes.byref(x), ctypes.byref(z), ctypes.byref(c), ctypes.byref(cap))
        K, W = batch.n_keys, batch.words
        counts = _tensor(batch, batch._counts_ptr, (batch.n_pairs,), "<i8")
        s.update(batch=batch, out={"counts": counts, "x": _tensor(batch, x.value, (K, W), "<i8"), "z": _tensor(batch, z.value, (K, W), "<i8"),
                                   "c": _tensor(batch, c.value, (K,), "<c16")})
    return s


def run(state):
    kind = state["kind"]
    if kind == "gradient":
        e = expectation(state["plan"], state["coeffs"], state["psi"])
        dc, dpsi = torch.autograd.grad(e, (state["coeffs"], state["psi"]))
        return {"value": e.detach(), "coeffs": dc, "psi": dpsi}
    if kind == "expect":
        e = state["op"].expectation_statevector(state["psi"])
        return [e.real, e.imag]
    if kind == "batch":
        b = state["batch"]
        b.replay()
        return {"values": b.values, "terms": b.term_values, "hpsi": b.hpsi}
    if kind == "matmul":
        return _terms(state["lhs"].matmul(state["rhs"], True, 1 << 31))
    if kind == "simplify":
        return _terms(state["op"].simplify())
    if kind == "flags":
        return torch.from_dlpack(state["lhs"].commutes_with_device(state["rhs"], 1 << 40))
    if kind == "bits":
        b = state["lhs"].commutes_with_bits(state["rhs"], 1 << 40)
        return _tensor(b, b.data_pointer, (b.shape[0], b.pitch_words), "<i4")
    if kind == "group":
        x, z = state["x"], state["z"]
        T, W = x.shape
        order, sizes, count = np.empty(T, np.uint64), np.zeros(T, np.uint64), ctypes.c_size_t()
        to = ctypes.POINTER(ctypes.c_size_t)
        capi.call("wg_group_commuting", x.device.index, W, T, x.data_ptr(), z.data_ptr(), int(state["case"]["full"]), order.ctypes.data_as(to),
                  sizes.ctypes.data_as(to), ctypes.byref(count), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return {"order": order.view(np.int64), "sizes": sizes.view(np.int64), "count": count.value}
    state["batch"].replay()
    return state["out"]


# ------------------------------------------------------------------ what a pass cannot do without


def _groups(n, T):
    """Distinct X parts: about T / 10 patterns, and no more than there are of weight 4 and below."""
    return min(max(4, T // 10), sum(math.comb(n, k) for k in range(min(4, n) + 1)))


def work(case):
    kind = case["kind"]
    amp = 8 if case.get("single") else 16
    if kind == "gradient":  # the state in, two values a term, the gradient out; a product a pair and a product an output
        N, T = 1 << case["qubits"], case["terms"]
        G = _groups(case["qubits"], T)
        return {"bytes": 2 * amp * N + 32 * T, "flops": G * N * (3 + 8)}
    if kind == "expect":
        N, T = 1 << case["qubits"], case["terms"]
        return {"bytes": amp * N + 32 * T, "flops": 3 * N * min(T, N)}
    if kind == "batch":
        r = _sizes(case)
        b = f = 0
        for _ in range(case["pairs"]):
            N = 1 << int(r.integers(case["low"], case["high"] + 1))
            T = int(round(math.exp(r.uniform(math.log(100), math.log(case["most"])))))
            b += (amp + 16) * N + 40 * T
            f += 11 * N * min(T, N)
        return {"bytes": b, "flops": f}
    if kind in ("flags", "bits"):
        W = (case["qubits"] + 63) // 64
        pairs = case["lhs"] * case["rhs"]
        return {"bytes": pairs / (1 if kind == "flags" else 8) + 16 * W * (case["lhs"] + case["rhs"]), "flops": 0}
    W = (case["qubits"] + 63) // 64
    if kind == "matmul":  # the operands in, the collected terms out: fewer than products where strings meet
        P = case["lhs"] * case["rhs"]
        out = min(P, 4.0 ** case["qubits"]) * (0.3 if case["family"] == "dense" else 0.9)
        return {"bytes": (16 * W + 16) * (case["lhs"] + case["rhs"] + out), "flops": 8 * P}
    if kind == "simplify":
        return {"bytes": (16 * W + 16) * (case["terms"] + case["distinct"]), "flops": 2 * case["terms"]}
    if kind == "group":
        return {"bytes": (16 * W + 8) * case["terms"], "flops": 0}
    r = _sizes(case)
    P = 0
    for _ in range(case["pairs"]):
        a, b = np.round(np.exp(r.uniform(math.log(case["low"]), math.log(case["high"]), size=2))).astype(int)
        P += int(a) * int(b)
    return {"bytes": (16 * W + 16) * 0.85 * P, "flops": 8 * P}


# ------------------------------------------------------------------ the same in plain torch, 64 bits


def _popcount(v):
    m = 0x5555555555555555
    v = v - ((v >> 1) & m)
    m = 0x3333333333333333
    v = (v & m) + ((v >> 2) & m)
    v = (v + (v >> 4)) & 0x0F0F0F0F0F0F0F0F
    return ((v * 0x0101010101010101) >> 56) & 0xFF


def _signs(z, lo, bits):
    """(2^bits, K) of (-1)^popcount(z & b) for the bits lo.. of z."""
    b = torch.arange(1 << bits, device=z.device)
    return 1.0 - 2.0 * (_popcount(b[:, None] & (z[None, :] >> lo) & ((1 << bits) - 1)) & 1).to(torch.float64)


def _expectation_exact(n, x, z, c, psi, want_h=True):
    x, z, psi = x[:, 0], z[:, 0], psi.to(torch.complex128)
    lo = n // 2
    y = _popcount(x & z) & 3
    phase = torch.tensor([1, 1j, -1, -1j], device=_DEV, dtype=torch.complex128)[y]
    at = torch.arange(1 << n, device=_DEV)
    e = torch.zeros(x.numel(), dtype=torch.float64, device=_DEV)
    h = torch.zeros(1 << n, dtype=torch.complex128, device=_DEV) if want_h else None
    order = torch.argsort(x, stable=True)
    values, counts = torch.unique_consecutive(x[order], return_counts=True)
    begin = 0
    for xv, k in zip(values.tolist(), counts.tolist()):
        own = order[begin : begin + k]
        begin += k
        other = at ^ xv
        up, down = _signs(z[own], lo, n - lo), _signs(z[own], 0, lo)
        t = (psi[other].conj() * psi).reshape(1 << (n - lo), 1 << lo)
        s = torch.complex(((t.real @ down) * up).sum(0), ((t.imag @ down) * up).sum(0))
        e[own] = (s * phase[own]).real
        if want_h:
            d = (c[own] * phase[own])
            f = torch.complex((up * d.real) @ down.T, (up * d.imag) @ down.T).reshape(-1)
            h += (f * psi)[other]
    return (c * e).sum(), e, h


def _collected(keys, c, cut=1e-12):
    """Words (most significant first) and coefficients of a sum, equal words collected, in order."""
    order = torch.arange(c.numel(), device=_DEV)
    top = -(1 << 63)
    for k in reversed(keys):
        order = order[torch.sort((k ^ top)[order], stable=True).indices]
    keys = [k[order] for k in keys]
    head = torch.ones(c.numel(), dtype=torch.bool, device=_DEV)
    head[1:] = False
    for k in keys:
        head[1:] |= k[1:] != k[:-1]
    seg = head.cumsum(0) - 1
    s = torch.zeros(int(seg[-1]) + 1, 2, dtype=torch.float64, device=_DEV)
    s.index_add_(0, seg, torch.view_as_real(c[order].contiguous()))
    s = torch.view_as_complex(s)
    return s[s.abs() > cut]


def _product_exact(l, r):
    (lx, lz, lc), (rx, rz, rc) = l, r
    keys, e = [], torch.zeros(lc.numel() * rc.numel(), dtype=torch.int64, device=_DEV)
    for w in range(lx.shape[1]):
        a, b, p, q = lx[:, w], lz[:, w], rx[:, w], rz[:, w]
        x, z = (a[:, None] ^ p[None, :]).reshape(-1), (b[:, None] ^ q[None, :]).reshape(-1)
        e += _popcount(x & z) + (2 * _popcount(a[:, None] & q[None, :]) - _popcount(a & b)[:, None] - _popcount(p & q)[None, :]).reshape(-1)
        keys += [x, z]
    c = (lc[:, None] * rc[None, :]).reshape(-1) * torch.tensor([1, 1j, -1, -1j], device=_DEV, dtype=torch.complex128)[e & 3]
    return _collected(keys, c)


def exact(case, seed):
    kind, n = case["kind"], case.get("qubits")
    if kind == "gradient":
        x, z, c, psi = _gradient_inputs(case, seed)
        value, e, h = _expectation_exact(n, x, z, c, psi)
        return {"value": value.real, "coeffs": e, "psi": 2.0 * h}
    if kind == "expect":
        x, z, c, psi = _expect_inputs(case, seed)
        value = complex(_expectation_exact(n, x, z, c, psi, want_h=False)[0])
        return [value.real, value.imag]
    if kind == "batch":
        out = {"values": [], "terms": [], "hpsi": []}
        for n, x, z, c, psi in _batch_inputs(case, seed):
            value, e, h = _expectation_exact(n, x, z, c, psi)
            out["values"].append(torch.view_as_real(value))
            out["terms"].append(e)
            out["hpsi"].append(h)
        return dict(out, values=torch.stack(out["values"]))
    if kind == "matmul":
        l, r = _matmul_inputs(case, seed)
        return {"x": None, "z": None, "c": _product_exact(l, r)}
    if kind == "simplify":
        x, z, c = _simplify_inputs(case, seed)
        keys = [k for w in range(x.shape[1]) for k in (x[:, w], z[:, w])]
        return {"x": None, "z": None, "c": _collected(keys, c)}
    if kind == "products":
        pairs = _products_inputs(case, seed)
        return {"counts": None, "x": None, "z": None, "c": torch.cat([_product_exact(a[1:], b[1:]) for a, b in pairs])}
    return None
