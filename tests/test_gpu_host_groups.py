"""Host products on either side of the operand size from which b goes up in column groups (7 MiB: 28 limbs
at N = 2^16), on both engines and with residues on the integer pipes, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import negacyclic as nc
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,bits", [(8192, 434), (32768, 1024), (65536, 864), (65536, 868)])
def test_upload_groups(gpu, N, bits):
    c = cases.make_case(N, bits, seed=N + bits, edge_frac=0.01)
    want = oracle.negacyclic(N, c.q_limbs, c.a, c.b)
    with nc.Plan(N, c.q_limbs) as plan:
        for _ in range(2):
            assert np.array_equal(plan.multiply(c.a, c.b), want)
        plan.word_bits = 64
        assert np.array_equal(plan.multiply(c.a, c.b), want)
        plan.residue_engine = nc.RESIDUES_IMAD
        assert np.array_equal(plan.multiply(c.a, c.b), want)
