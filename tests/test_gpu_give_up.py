"""A kernel's bounded wait that runs out is reported (NC_ETIMEOUT), by each kernel that waits on a copy or
on MMAs, and the context stays usable. The library's test build counts waits as run out once they are
over (NC_GIVE_UP, read at each launch: 1 tables, 2 MMAs, 4 the blocks of the 30-bit rows), so nothing is left in flight. One process a
setting, on that build."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("give_up", [1, 2, 4])
@pytest.mark.parametrize("what", ["product", "batch"])
def test_run_out_wait_is_reported(gpu, give_up, what):
    r = subprocess.run([sys.executable, __file__, what, str(give_up)], timeout=600, capture_output=True, text=True)
    assert r.returncode == 0 and "reported" in r.stdout, r.stdout + r.stderr


def _main(what: str, give_up: str) -> None:
    import conftest  # noqa: F401  (import paths)
    import numpy as np
    import torch

    import cases
    import negacyclic as nc
    import oracle

    nc.LIB_PATH = nc.LIB_PATH.with_name("libnegacyclic_b200_give_up.so")

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).cuda()

    def reports(fn):
        os.environ["NC_GIVE_UP"] = give_up
        try:
            for _ in range(2):  # the call itself, and every later one
                try:
                    fn()
                except nc.NegacyclicError as e:
                    assert e.code == nc.NC_ETIMEOUT, e
                else:
                    raise AssertionError("not reported")
                os.environ.pop("NC_GIVE_UP", None)
        finally:
            os.environ.pop("NC_GIVE_UP", None)

    # one pass of 32 (30-bit) or 16 (62-bit) primes and more, fewer coefficients than a tile, 32-point columns;
    # beyond 32 primes of the 62-bit engine its CRT has no MMAs
    for N, bits, word in [(8, 127, None), (256, 868, None), (4096, 434, None), (65536, 868, None), (8, 127, 64),
                          (4096, 868, 64), (4096, 1000, 64), (65536, 434, 64), (2, 100, None), (4, 300, None),
                          (8192, 600, None)]:
        if give_up == "4" and word == 64:
            continue  # the 62-bit rows wait on nothing
        c = cases.make_case(N, bits, seed=3 * N + bits, edge_frac=0.02)
        want = oracle.negacyclic(N, c.q_limbs, c.a, c.b)
        with nc.Plan(N, c.q_limbs, word_bits=word) as plan:
            if what == "product":
                assert np.array_equal(plan.multiply(c.a, c.b), want)
                reports(lambda: plan.multiply(c.a, c.b))
            else:
                a, b = dev(c.a), dev(c.b)
                out = torch.full_like(a, -1)
                with nc.Batch() as batch:
                    batch.add(plan, a.data_ptr(), b.data_ptr(), out.data_ptr())

                    def run():
                        batch.run(0, False)
                        batch.synchronize()

                    run()
                    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
                    reports(run)
        # with its last plan the device's tables go, and a new plan's products are good again
    print("reported")


if __name__ == "__main__":
    _main(*sys.argv[1:])
