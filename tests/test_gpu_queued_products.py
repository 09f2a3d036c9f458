"""Products queued back to back on one plan without a wait between them, so that each kernel may be
scheduled while the one before it runs: every output against the oracle, at the ring degrees and prime
counts on either side of the 30-bit engine's rule for releasing the next kernel early (N = 32 and 64; 16 and 17
primes from N = 2^14)."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import negacyclic as nc
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,bits", [(2, 100), (8, 868), (16, 100), (32, 434), (64, 434), (8192, 200), (16384, 31),
                                    (16384, 225), (16384, 245), (32768, 130), (65536, 100), (65536, 300)])
def test_queued_products(gpu, N, bits):
    import torch

    c = cases.make_case(N, bits, seed=13 * N + bits, edge_frac=0.01)
    d = cases.make_case(N, bits, seed=17 * N + bits, edge_frac=0.01, q=c.q)
    ops = [torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).to(gpu) for x in (c.a, c.b, d.a, d.b)]
    pairs = [(0, 1), (2, 3), (0, 3), (1, 2)]
    host = (c.a, c.b, d.a, d.b)
    want = [oracle.negacyclic(N, c.q_limbs, host[i], host[j]) for i, j in pairs]
    with nc.Plan(N, c.q_limbs, word_bits=32) as plan:
        outs = [torch.full_like(ops[0], -1) for _ in range(24)]
        torch.cuda.synchronize()
        for r, out in enumerate(outs):
            i, j = pairs[r % 4]
            plan.multiply_device(ops[i].data_ptr(), ops[j].data_ptr(), out.data_ptr(), 0)
        torch.cuda.synchronize()
        for r, out in enumerate(outs):
            assert np.array_equal(out.cpu().numpy().view(np.uint32), want[r % 4]), (r, plan.plain_primes)
