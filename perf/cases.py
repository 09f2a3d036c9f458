"""Cases that time the library through its Python entry points.

A case is a plain dict: `kind` names the entry point (below), `N` the ring degree, `bits` the width
of the modulus, `count` the products of a batch or the operands of a chain, `tune` whether the
program runs the plan's autotuner first (as fherma_init does), `edge` the share of coefficients
that are 0, 1, q - 1 or a power of two. The modulus of a width is one seeded prime, as a deployed
ring has; the coefficients come from the seed.

    device   Plan.multiply_device                 one product, operands on the GPU
    noalloc  Plan.multiply_device_noalloc         the same for callers that own the GPU's memory
    chain    Plan.multiply_chain_device           x_0 x_1 .. x_{count-1} with one reduction
    batch    Batch of `count` equal products      one captured graph, replayed
    mix      Batch of `count` uneven products     N over 2^10 .. N, 434- and 868-bit moduli
    cached   Batch.add_forward of 8 operands, then `count` Batch.add_cached products on them
    host     Plan.multiply on host arrays         uploads, product and download in the call
"""
from __future__ import annotations

import functools
import importlib
import math
import random

import numpy as np
import torch

_PACKAGE = "engel-cuda-negacyclic-multiply_b200"
nc = importlib.import_module(_PACKAGE + ".negacyclic")
_gen = importlib.import_module(_PACKAGE + ".cases")

RESIDENT = 8  # operands kept in the NTT domain by a `cached` case


def listed():
    return [
        # the smallest ring of the reference's points: launches and latency decide
        {"name": "device_n1024_q868", "kind": "device", "N": 1024, "bits": 868, "count": 1, "tune": False, "edge": 0.0},
        # a latency-critical loop that may not allocate
        {"name": "noalloc_n2048_q434", "kind": "noalloc", "N": 2048, "bits": 434, "count": 1, "tune": False, "edge": 0.0},
        # an odd limb count (19), so no limb row is aligned
        {"name": "device_n4096_q600", "kind": "device", "N": 4096, "bits": 600, "count": 1, "tune": False, "edge": 0.01},
        # an ordinary single product
        {"name": "device_n16384_q868", "kind": "device", "N": 16384, "bits": 868, "count": 1, "tune": True, "edge": 0.0},
        # the headline product, with its 1% of edge values
        {"name": "device_n65536_q868", "kind": "device", "N": 65536, "bits": 868, "count": 1, "tune": True, "edge": 0.01},
        # the widest moduli, beyond 64 thirty-bit primes
        {"name": "device_n65536_q1000", "kind": "device", "N": 65536, "bits": 1000, "count": 1, "tune": False, "edge": 0.01},
        # a product of three operands with one reduction
        {"name": "chain3_n16384_q868", "kind": "chain", "N": 16384, "bits": 868, "count": 3, "tune": False, "edge": 0.0},
        # the uniform batch of the benchmark
        {"name": "batch64_n16384_q868", "kind": "batch", "N": 16384, "bits": 868, "count": 64, "tune": False, "edge": 0.0},
        # the benchmark's uneven mix, what a server's batches look like
        {"name": "mix256_n65536", "kind": "mix", "N": 65536, "bits": 868, "count": 256, "tune": False, "edge": 0.0},
        # resident operands: transformed once, then used by several products
        {"name": "cached32_n4096_q868", "kind": "cached", "N": 4096, "bits": 868, "count": 32, "tune": False, "edge": 0.0},
        # the drop-in call on host vectors, a middling and the headline size
        {"name": "host_n8192_q434", "kind": "host", "N": 8192, "bits": 434, "count": 1, "tune": False, "edge": 0.0},
        {"name": "host_n65536_q868", "kind": "host", "N": 65536, "bits": 868, "count": 1, "tune": True, "edge": 0.01},
    ]


def draw(rng):
    kind = rng.choice(["device", "device", "device", "noalloc", "chain", "batch", "batch", "mix", "cached", "host"])
    top = {"noalloc": 14, "mix": 14, "cached": 14}.get(kind, 16)
    log_n = rng.randint(10, top)
    # any width: the usual ones and arbitrary ones between 64 bits and the widest modulus
    bits = rng.choice([434, 868, rng.randint(64, 1020), rng.randint(64, 1020)])
    count = 1
    if kind == "noalloc" and log_n == 14:
        bits = min(bits, 868)  # the limit of the library's fixed scratch
    elif kind == "chain":
        count = rng.randint(3, 4)
        bits = min(bits, 868 if count == 3 else 700)
    elif kind in ("batch", "cached"):
        count = max(2, int(2 ** rng.uniform(1, min(7, 19 - log_n))))
    elif kind == "mix":
        count = rng.randint(8, 160)
    return {"kind": kind, "N": 1 << log_n, "bits": bits, "count": count, "tune": rng.random() < 0.5,
            "edge": rng.choice([0.0, 0.01])}


@functools.lru_cache(maxsize=None)
def _modulus(bits):
    return _gen.gen_prime_fast(bits, 1000 + bits)


def _q(bits):
    L = (bits + 31) // 32
    return _gen.limbs_of(_modulus(bits), L), L


def _shapes(case):
    """(N, bits) of every product of the case."""
    if case["kind"] != "mix":
        return [(case["N"], case["bits"])] * (1 if case["kind"] == "chain" else case["count"])
    rng = random.Random(case["count"])
    hi = case["N"].bit_length() - 1
    return [(1 << rng.randint(10, hi), rng.choice([434, 868])) for _ in range(case["count"])]


def _coeffs(n, bits, edge, gen):
    """(n, L) limbs on the GPU, uniform below the modulus's leading limb, a share of them edge values."""
    q, L = _q(bits)
    x = torch.randint(-(1 << 31), 1 << 31, (n, L), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    top = torch.randint(0, int(q[-1]), (n,), generator=gen, device="cuda", dtype=torch.int64)
    x[:, -1] = torch.where(top >= 1 << 31, top - (1 << 32), top).to(torch.int32)
    n_edge = int(round(n * edge))
    if n_edge:
        values = [0, 1, _modulus(bits) - 1] + [pow(2, k, _modulus(bits)) for k in (31, 32, 100, bits - 1, bits + 31)]
        table = torch.from_numpy(_gen.rows_of_ints(values, L).view(np.int32)).cuda()
        pick = torch.randint(0, len(values), (n_edge,), generator=gen, device="cuda")
        where = torch.randperm(n, generator=gen, device="cuda")[:n_edge]
        x[where] = table[pick]
    return x


def _operands(case, seed):
    """The case's operands on the GPU: a list of tuples, one for each product (a chain's is its x)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    N, bits, edge = case["N"], case["bits"], case["edge"]
    if case["kind"] == "chain":
        return [tuple(_coeffs(N, bits, edge, gen) for _ in range(case["count"]))]
    if case["kind"] == "cached":
        a = [_coeffs(N, bits, edge, gen) for _ in range(RESIDENT)]
        return [(a[i % RESIDENT], _coeffs(N, bits, edge, gen)) for i in range(case["count"])]
    return [(_coeffs(n, w, edge, gen), _coeffs(n, w, edge, gen)) for n, w in _shapes(case)]


def prepare(case, seed):
    kind = case["kind"]
    ops = _operands(case, seed)
    shapes = _shapes(case)
    plans = {}
    for n, bits in shapes:
        if (n, bits) not in plans:
            plans[n, bits] = nc.Plan(n, _q(bits)[0], factors=case["count"] if kind == "chain" else 2)
            if case["tune"]:
                plans[n, bits].autotune()
    state = {"case": case, "plans": plans, "ops": ops, "plan": plans[shapes[0]]}
    if kind == "host":
        state["host"] = tuple(x.cpu().numpy().view(np.uint32) for x in ops[0])
        state["out"] = np.zeros_like(state["host"][0])
        return state
    # one buffer for all products, each a slice of it
    sizes = [n * ((bits + 31) // 32) for n, bits in shapes]
    out = torch.zeros(sum(sizes), dtype=torch.int32, device="cuda")
    at = [sum(sizes[:i]) for i in range(len(sizes))]
    state["out"] = out
    state["c"] = [out[i:i + s].data_ptr() for i, s in zip(at, sizes)]
    state["ptrs"] = [tuple(x.data_ptr() for x in t) for t in ops]
    if kind in ("batch", "mix"):
        state["batch"] = nc.Batch()
        for (n, bits), (a, b), c in zip(shapes, state["ptrs"], state["c"]):
            state["batch"].add(plans[n, bits], a, b, c)
    elif kind == "cached":
        plan = state["plan"]
        hats = torch.empty((RESIDENT, plan.hat_words), dtype=torch.int64, device="cuda")
        state["hats"], state["forward"], state["batch"] = hats, nc.Batch(), nc.Batch()
        for i in range(min(RESIDENT, case["count"])):
            state["forward"].add_forward(plan, state["ptrs"][i][0], hats[i].data_ptr())
        for i, ((_, b), c) in enumerate(zip(state["ptrs"], state["c"])):
            state["batch"].add_cached(plan, hats[i % RESIDENT].data_ptr(), b, c)
    return state


def run(state):
    kind, plan = state["case"]["kind"], state["plan"]
    if kind == "host":
        a, b = state["host"]
        return plan.multiply(a, b, out=state["out"])
    if kind == "device":
        plan.multiply_device(*state["ptrs"][0], state["c"][0])
    elif kind == "noalloc":
        plan.multiply_device_noalloc(*state["ptrs"][0], state["c"][0])
    elif kind == "chain":
        plan.multiply_chain_device(state["ptrs"][0], state["c"][0])
    else:
        if kind == "cached":
            state["forward"].run()
        state["batch"].run()
    return state["out"]


def work(case):
    """Operands read and products written once; the multiply-adds (two operations each) of residues
    modulo 30-bit primes, their transforms and the recombination."""
    total = {"bytes": 0, "flops": 0}
    operands = case["count"] if case["kind"] == "chain" else 2
    for n, bits in _shapes(case):
        L, log_n = (bits + 31) // 32, n.bit_length() - 1
        k = math.ceil((operands * bits + (operands - 1) * log_n) / 30)
        total["bytes"] += (operands + 1) * n * L * 4
        total["flops"] += 2 * k * n * ((operands + 1) * log_n // 2 + (operands + 1) * L)
    return total


def _product(a, b, bits):
    """a b mod (X^N + 1, q) of (N, L) limbs: an FFT of bytes in 64-bit floats (every sum of byte products
    is below 2^39, so it rounds to the integer), then exact integers."""
    q, L = _q(bits)
    n, d = a.shape[0], 4 * L
    twist = np.exp(1j * np.pi * np.arange(n) / n)[:, None]
    f = [np.fft.fft2(np.ascontiguousarray(x).view(np.uint8).reshape(n, d) * twist, s=(n, 2 * d)) for x in (a, b)]
    s = np.rint((np.fft.ifft2(f[0] * f[1]) * np.conj(twist)).real).astype(np.int64)
    digits, carry = np.zeros((n, 2 * d + 8), dtype=np.uint8), np.zeros(n, dtype=np.int64)
    for i in range(2 * d + 8):
        t = carry + (s[:, i] if i < 2 * d else 0)
        digits[:, i], carry = t & 255, t >> 8
    m, top = _modulus(bits), 1 << (8 * (2 * d + 8))
    rows = [(int.from_bytes(digits[i].tobytes(), "little") + int(carry[i]) * top) % m for i in range(n)]
    return _gen.rows_of_ints(rows, L)


def exact(case, seed):
    """The products as exact integers; None where that takes too long here."""
    shapes = _shapes(case)
    if sum(n for n, _ in shapes) * (case["count"] - 1 if case["kind"] == "chain" else 1) > 1 << 17:
        return None
    out = []
    for (_, bits), t in zip(shapes, _operands(case, seed)):
        t = [x.cpu().numpy().view(np.uint32) for x in t]
        c = t[0]
        for x in t[1:]:
            c = _product(c, x, bits)
        out.append(c)
    return out[0] if case["kind"] == "host" else np.concatenate([c.reshape(-1) for c in out]).view(np.int32)
