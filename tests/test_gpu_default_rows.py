"""The 62-bit engine's default row shape follows the residue engine where the two differ (N = 2^16, up to
18 primes), a shape that the caller set stays, and products are the oracle's throughout."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import negacyclic as nc
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,bits,imad", [(65536, 530, (12, 3, 512)), (65536, 560, (11, 3, 256)),
                                         (32768, 434, (11, 3, 256))])
def test_default_shape_follows_the_residue_engine(gpu, N, bits, imad):
    c = cases.make_case(N, bits, seed=N + bits, edge_frac=0.01)
    want = oracle.negacyclic(N, c.q_limbs, c.a, c.b)
    with nc.Plan(N, c.q_limbs, word_bits=64) as plan:
        assert plan.row_config == (11, 3, 256)
        plan.residue_engine = nc.RESIDUES_IMAD
        assert plan.row_config == imad
        assert np.array_equal(plan.multiply(c.a, c.b), want)
        plan.residue_engine = nc.RESIDUES_TC_I8
        assert plan.row_config == (11, 3, 256)
        assert np.array_equal(plan.multiply(c.a, c.b), want)
        plan.row_config = (12, 4, 256)
        plan.residue_engine = nc.RESIDUES_IMAD
        assert plan.row_config == (12, 4, 256)
        assert np.array_equal(plan.multiply(c.a, c.b), want)
