"""Every compiled row shape of the 30-bit engine at the ring degrees whose blocks have an uneven last
pass or a padded place per residue (2^2 to 2^5 points, 2^7 to 2^9, 2^11, 2^15), alone and in a batch's
persistent rows, against the oracle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import negacyclic as nc
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n", [2, 3, 4, 5, 7, 8, 9, 11, 15])
def test_row_shapes(gpu, log_n):
    import torch

    N = 1 << log_n
    c = cases.make_case(N, 868, seed=700 + log_n, edge_frac=0.02)
    want = oracle.negacyclic(N, c.q_limbs, c.a, c.b)
    a, b = (torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).to(gpu) for x in (c.a, c.b))
    with nc.Plan(N, c.q_limbs, word_bits=32) as plan:
        for cfg in nc.row_variants(log_n, word_bits=32):
            plan.row_config = cfg
            assert np.array_equal(plan.multiply(c.a, c.b), want), cfg
            batch = nc.Batch()
            outs = [torch.empty_like(a) for _ in range(3)]
            for out in outs:
                batch.add(plan, a.data_ptr(), b.data_ptr(), out.data_ptr())
            batch.run(0, True)
            for out in outs:
                assert np.array_equal(out.cpu().numpy().view(np.uint32), want), (cfg, "batch")
