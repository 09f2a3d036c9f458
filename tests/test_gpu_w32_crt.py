"""The 30-bit engine's CRT where its one-word quotient and its tiles have edges, bit for bit against
the oracle: moduli from 3 bits up whose leading byte is full, barely begun or at a limb's end (the
quotient reads five bytes from the leading one down), every limb-count class, and the ring degrees on
either side of a change of tile."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import negacyclic as nc
import oracle

pytestmark = pytest.mark.gpu


def check(N, q, seed):
    L = (q.bit_length() + 31) // 32
    ql = cases.limbs_of(q, L)
    a, b = cases.coeffs(q, N, L, seed, 0.05), cases.coeffs(q, N, L, seed + 1, 0.05)
    top = np.tile(cases.limbs_of(q - 1, L), (N, 1))
    with nc.Plan(N, ql, word_bits=32) as plan:
        for x, y in ((a, b), (top, top), (top, b)):
            assert np.array_equal(plan.multiply(x, y), oracle.negacyclic(N, ql, x, y)), (N, q.bit_length())


@pytest.mark.parametrize("bits", [3, 8, 13, 14, 15, 32, 33, 39, 40, 41, 47, 64, 65, 72, 96, 97, 104, 127, 128, 129, 223,
                                  255, 256, 257, 480, 481, 511, 512, 513, 640, 767, 896, 897, 928, 929, 947])
def test_quotient_at_every_alignment(gpu, bits):
    """The largest and the smallest odd modulus of the width (composite moduli are accepted)."""
    for q in ((1 << bits) - 1, (1 << (bits - 1)) + 1):
        check(64, q, 7 * bits)


@pytest.mark.parametrize("log_n", [1, 4, 5, 6, 7, 8, 10, 11, 12, 13, 14, 15])
@pytest.mark.parametrize("bits", [100, 434, 600])
def test_tiles(gpu, log_n, bits):
    check(1 << log_n, cases.gen_prime(bits, 31), 3 * log_n + bits)
