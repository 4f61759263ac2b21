"""Batches of different shared-memory needs solved from two threads at once: neither's set-up takes the other's launches
their shared memory."""
import threading

import numpy as np
import pytest

from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G

pytestmark = pytest.mark.gpu

GENERAL = dict(ctaKernel=_lib.CTA_GENERAL, ctaThreads=256)


@pytest.mark.parametrize("precision,large,small", [
    (_lib.PRECISION_FP64, GENERAL, GENERAL),
    (_lib.PRECISION_MIXED, GENERAL, GENERAL),
    (_lib.PRECISION_FP64, dict(ctaKernel=_lib.CTA_OWNER2, ctaThreads=512),
     dict(ctaKernel=_lib.CTA_OWNER2, ctaThreads=512)),
    (_lib.PRECISION_FP64, dict(ctaKernel=_lib.CTA_SLAB4), dict(ctaKernel=_lib.CTA_SLAB4, ctaSmemLimit=20_000)),
])
def test_two_needs(precision, large, small):
    def solve(lps, o):
        return pdhg.solvePdhgMulti(lps, pdhg.PdhgOptions(tolerance=1e-30, maxIterations=50, precision=precision,
                                                         multiForm=_lib.MULTI_CTA, **o))

    jobs = [([G.random_lp(500, 900, 5.0, 200, 71 + i) for i in range(4)], large),
            ([G.random_lp(20, 30, 3.0, 9, 75 + i) for i in range(4)], small)]
    want = [solve(*j) for j in jobs]
    failed = []

    def work(q):
        try:
            for _ in range(60):
                for a, b in zip(solve(*jobs[q]), want[q]):
                    if not (np.array_equal(a.x, b.x) and np.array_equal(a.rowDual, b.rowDual)):
                        failed.append((q, "another answer"))
        except Exception as e:
            failed.append((q, repr(e)))

    threads = [threading.Thread(target=work, args=(q,)) for q in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
