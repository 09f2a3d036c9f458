"""nc_multiply_device_noalloc on either engine, bit for bit against the oracle: the 30-bit engine's
residues of the largest product that the fixed scratch admits, the smallest, and a modulus beyond it."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import negacyclic as nc
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,bits,word", [(2, 100, None), (2048, 434, None), (2048, 434, 64), (16384, 868, None),
                                         (16384, 868, 64), (32768, 434, None), (8192, 1000, None)])
def test_noalloc_engines(gpu, N, bits, word):
    import torch

    c = cases.make_case(N, bits, seed=77 + N + bits, edge_frac=0.02)
    with nc.Plan(N, c.q_limbs, word_bits=word) as plan:
        a, b = (torch.from_numpy(x.view(np.int32)).to(gpu) for x in (c.a, c.b))
        out = torch.full_like(a, -1)
        plan.multiply_device_noalloc(a.data_ptr(), b.data_ptr(), out.data_ptr(), 0)
        torch.cuda.synchronize()
        got = out.cpu().numpy().view(np.uint32).reshape(N, c.L)
    assert np.array_equal(got, oracle.negacyclic(N, c.q_limbs, c.a, c.b))
