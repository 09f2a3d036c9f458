"""The 30-bit row kernels in product mode (multiply_device, which autotuning times too), every compiled shape
at every ring degree; and a batch's persistent rows, mirror pairs of blocks among them (2^12 to 2^14), with
products, forward and cached items. Outputs hold -1 before each run; all bit for bit against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import negacyclic as nc
import oracle

pytestmark = pytest.mark.gpu


def _dev(x, gpu):
    import torch

    return torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).to(gpu)


@pytest.mark.parametrize("log_n", range(1, 17))
@pytest.mark.parametrize("bits", [100, 868])
def test_every_shape_in_product_mode(gpu, log_n, bits):
    N = 1 << log_n
    c = cases.make_case(N, bits, seed=1700 + 20 * log_n + bits, edge_frac=0.02)
    want = oracle.negacyclic(N, c.q_limbs, c.a, c.b)
    a, b = _dev(c.a, gpu), _dev(c.b, gpu)
    out = a.clone()
    with nc.Plan(N, c.q_limbs, word_bits=32) as plan:
        for cfg in nc.row_variants(log_n, word_bits=32):
            plan.row_config = cfg
            out.fill_(-1)
            plan.multiply_device(a.data_ptr(), b.data_ptr(), out.data_ptr(), 0)
            assert np.array_equal(out.cpu().numpy().view(np.uint32), want), cfg


@pytest.mark.parametrize("log_n", range(1, 17))
@pytest.mark.parametrize("bits", [100, 868])
def test_batch_rows_in_every_mode(gpu, log_n, bits):
    import torch

    N = 1 << log_n
    c = cases.make_case(N, bits, seed=2700 + 20 * log_n + bits, edge_frac=0.02)
    want = oracle.negacyclic(N, c.q_limbs, c.a, c.b)
    square = oracle.negacyclic(N, c.q_limbs, c.b, c.b)
    a, b = _dev(c.a, gpu), _dev(c.b, gpu)
    outs = [a.clone() for _ in range(4)]
    with nc.Plan(N, c.q_limbs, word_bits=32) as plan, nc.Batch() as forward, nc.Batch() as batch:
        hat = torch.full((plan.hat_words,), -1, dtype=torch.int64, device=gpu)
        forward.add_forward(plan, a.data_ptr(), hat.data_ptr())
        forward.run(0, True)
        forward.synchronize()
        batch.add(plan, a.data_ptr(), b.data_ptr(), outs[0].data_ptr())
        batch.add_cached(plan, hat.data_ptr(), b.data_ptr(), outs[1].data_ptr())
        batch.add(plan, b.data_ptr(), b.data_ptr(), outs[2].data_ptr())
        batch.add(plan, b.data_ptr(), a.data_ptr(), outs[3].data_ptr())
        for _ in range(2):
            for out in outs:
                out.fill_(-1)
            batch.run(0, True)
            batch.synchronize()
            for out, expected in zip(outs, (want, want, square, want)):
                assert np.array_equal(out.cpu().numpy().view(np.uint32), expected)
