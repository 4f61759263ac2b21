"""The CTA form's kernel variants: every one gives the same answers bit for bit, checks, restarts and all, since a
check's sums have one order whatever the threads; the choice is made per precision; a deadline still stops a run."""
import threading
import time

import ctypes as C
import numpy as np
import pytest

from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G

pytestmark = pytest.mark.gpu


def _same(a, b):
    return (np.array_equal(a.x, b.x) and np.array_equal(a.rowDual, b.rowDual) and a.objective == b.objective
            and a.relativeKkt == b.relativeKkt and a.iterations == b.iterations and a.status == b.status)


@pytest.mark.parametrize("sizes", [(1, 31, 33), (127, 129, 255), (257, 511, 400), (513, 700, 1025)])
@pytest.mark.parametrize("precision", [_lib.PRECISION_FP64, _lib.PRECISION_MIXED])
def test_variants_agree(sizes, precision):
    lps = [G.random_lp(m, 2 * m, min(4.0, m), m // 2, 41 + m) for m in sizes]
    ref = None
    variants = [dict(ctaThreads=t, ctaKernel=_lib.CTA_GENERAL) for t in (128, 256, 512, 1024)]
    if precision == _lib.PRECISION_FP64:
        most = 2 * max(sizes)
        variants += [dict(ctaThreads=t, ctaKernel=k) for t in (128, 256, 512)
                     for r, k in ((1, _lib.CTA_OWNER1), (2, _lib.CTA_OWNER2)) if most <= t * r]
    variants.append(dict())
    for v in variants:
        res = pdhg.solvePdhgMulti(lps, pdhg.PdhgOptions(tolerance=1e-5, maxIterations=3000, precision=precision,
                                                        multiForm=_lib.MULTI_CTA, **v))
        ref = ref or res
        assert all(_same(a, b) for a, b in zip(res, ref)), v


def test_cancel_reaches_the_blocks():
    lps = [G.random_lp(100, 200, 4.0, 50, 42 + i) for i in range(300)]
    flag = (C.c_int32 * 1)(0)
    po = pdhg.PdhgOptions(tolerance=1e-30, maxIterations=200_000_000, multiForm=_lib.MULTI_CTA, timeLimit=20.0)
    threading.Timer(0.5, lambda: flag.__setitem__(0, 1)).start()
    t = time.perf_counter()
    res = pdhg.solvePdhgMulti(lps, po, cancel_flag=flag)
    assert time.perf_counter() - t < 10.0
    assert {r.status for r in res} == {"TimeLimit"}
