"""The kernels' bounded waits giving up (NC_GIVE_UP in the library's environment: 1, the first wait for
each copy; 4 beside it, a second wait counts as run out too): products stay bit for bit the oracle's
where the second wait ends, and are reported where it does not. Each setting runs in a process of its
own; every copy is waited for in all of them."""
from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# fewer coefficients than a tile, one pass of primes and two, limb counts that are odd and multiples of four
POINTS = [(2, 100), (64, 300), (256, 868), (2048, 434), (4096, 600), (16384, 868), (65536, 868), (4096, 1000)]


def run(give_up: int, what: str) -> str:
    r = subprocess.run([sys.executable, __file__, what], env=dict(os.environ, NC_GIVE_UP=str(give_up)), timeout=600,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.parametrize("give_up", [1])
@pytest.mark.parametrize("what", ["device", "batch", "chain"])
def test_results_stand(gpu, give_up, what):
    assert "same" in run(give_up, what)


def test_late_copy_is_reported(gpu):
    """The plan's own self-test product is the first to report; every later call on the device does."""
    assert "reported" in run(5, "report")


def _main(what: str) -> None:
    import conftest  # noqa: F401  (import paths)
    import torch

    import cases
    import negacyclic as nc
    import oracle

    if what == "report":
        for _ in range(2):
            try:
                nc.Plan(4096, cases.make_case(4096, 868, seed=1).q_limbs)
            except nc.NegacyclicError as e:
                assert e.code == nc.NC_ETIMEOUT, e
            else:
                raise AssertionError("not reported")
        assert int(torch.ones(8, device="cuda").sum()) == 8  # the context is as good as before
        print("reported")
        return

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).cuda()

    def same(t, want):
        return np.array_equal(t.cpu().numpy().view(np.uint32), want)

    if what == "chain":
        for N, bits in [(64, 434), (4096, 600), (16384, 868)]:
            c = cases.make_case(N, bits, seed=5 * N + bits, edge_frac=0.02)
            x = [c.a, c.b, c.a]
            want = oracle.negacyclic(N, c.q_limbs, oracle.negacyclic(N, c.q_limbs, c.a, c.b), c.a)
            d = [dev(v) for v in x]
            out = torch.full_like(d[0], -1)
            with nc.Plan(N, c.q_limbs, factors=3) as plan:
                plan.multiply_chain_device([v.data_ptr() for v in d], out.data_ptr(), 0)
                torch.cuda.synchronize()
                assert same(out, want), (N, bits)
        print("same")
        return
    keep = []
    batch = nc.Batch()
    for N, bits in POINTS:
        c = cases.make_case(N, bits, seed=3 * N + bits, edge_frac=0.02)
        want = oracle.negacyclic(N, c.q_limbs, c.a, c.b)
        for word in (None, 64):
            plan = nc.Plan(N, c.q_limbs, word_bits=word)
            a, b = dev(c.a), dev(c.b)
            out = torch.full_like(a, -1)
            if what == "device":
                for _ in range(2):
                    out.fill_(-1)
                    plan.multiply_device(a.data_ptr(), b.data_ptr(), out.data_ptr(), 0)
                    torch.cuda.synchronize()
                    assert same(out, want), (N, bits, word)
                assert np.array_equal(plan.multiply(c.a, c.b), want), (N, bits, word, "host")
                plan.close()
            else:
                batch.add(plan, a.data_ptr(), b.data_ptr(), out.data_ptr())
                hat = torch.zeros(plan.hat_words, dtype=torch.int64, device="cuda")
                with nc.Batch() as fwd:
                    fwd.add_forward(plan, a.data_ptr(), hat.data_ptr())
                    fwd.run(0, True)
                    fwd.synchronize()
                cached = torch.full_like(a, -1)
                batch.add_cached(plan, hat.data_ptr(), b.data_ptr(), cached.data_ptr())
                keep.append((plan, a, b, out, hat, cached, want, (N, bits, word)))
    if what == "batch":
        for _ in range(2):
            for item in keep:
                item[3].fill_(-1)
                item[5].fill_(-1)
            batch.run(0, True)
            batch.synchronize()
            for plan, a, b, out, hat, cached, want, at in keep:
                assert same(out, want), at
                assert same(cached, want), (at, "cached")
        batch.close()
    print("same")


if __name__ == "__main__":
    _main(sys.argv[1])
