"""The slab kernel (one LP per cluster of 2, 4 or 8 blocks): the general kernel's answers bit for bit, for a family that
shares its operator and for LPs with their own, in both precisions, at sizes around one slice (32), one round of a
block's warps and the largest that fit; and through a deadline."""
import numpy as np
import pytest

from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G
from pramana_b200 import warmstart as W

pytestmark = pytest.mark.gpu


def _check(lps, threads, iters, tol=1e-30, precision=_lib.PRECISION_FP64, starts=None):
    po = dict(tolerance=tol, maxIterations=iters, precision=precision, multiForm=_lib.MULTI_CTA)
    got = pdhg.solvePdhgMulti(lps, pdhg.PdhgOptions(ctaThreads=threads, **po), starts=starts)
    want = pdhg.solvePdhgMulti(lps, pdhg.PdhgOptions(ctaThreads=256, ctaKernel=_lib.CTA_GENERAL, **po), starts=starts)
    for a, b in zip(got, want):
        assert np.array_equal(a.x, b.x) and np.array_equal(a.rowDual, b.rowDual)
        assert (a.status, a.iterations, a.objective, a.relativeKkt) == (b.status, b.iterations, b.objective,
                                                                        b.relativeKkt)


# one block cannot hold the operators of any of these (LPs that fit do not take the slab kernel): 14,000 entries and
# more; 3,585 columns are one slice more than 2 blocks of 512 threads hold at two slices a warp
@pytest.mark.parametrize("m,n,per", [(500, 2800, 5.0), (33, 3000, 5.0), (1700, 3584, 4.0), (1700, 3585, 4.0),
                                     (1025, 4097, 4.0), (2049, 2000, 8.0)])
@pytest.mark.parametrize("threads", [0, 512, 1024])
@pytest.mark.parametrize("precision", [_lib.PRECISION_FP64, _lib.PRECISION_MIXED])
def test_own_operators(m, n, per, threads, precision):
    lps = [G.random_lp(m, n, min(per, m), m // 2, 51 + i) for i in range(2)] + [G.random_lp(20, 30, 3.0, 9, 50)]
    _check(lps, threads, 200, precision=precision)


@pytest.mark.parametrize("threads", [0, 512, 1024])
@pytest.mark.parametrize("precision", [_lib.PRECISION_FP64, _lib.PRECISION_MIXED])
def test_family_to_tolerance(threads, precision):
    fam = W.RefineryFamily(seed=5, periods=6, regions=2, units=6, streams=6, properties=3, pools=12,
                           scale_exponent=0.0)
    lps = [fam.instance(p) for p in fam.sample(5, seed=52)]
    rng = np.random.default_rng(53)
    starts = [(rng.uniform(0, 10, size=lps[0].num_cols), rng.standard_normal(lps[0].num_rows)), None, (None, None),
              None, None]
    _check(lps, threads, 3000, tol=1e-3, precision=precision, starts=starts)


def test_deadline():
    lps = [G.random_lp(1700, 3500, 4.0, 800, 54 + i) for i in range(3)]
    res = pdhg.solvePdhgMulti(lps, pdhg.PdhgOptions(tolerance=1e-30, maxIterations=200_000_000, timeLimit=0.5,
                                                    multiForm=_lib.MULTI_CTA))
    assert {r.status for r in res} == {"TimeLimit"}


def test_choice_of_another_batch_of_the_same_shape():
    """A batch with the sizes of an earlier one that the slab kernel cannot hold: one row of 2,500 entries, whose slice
    of 32 rows would be 800 KB."""
    m, n, per = 1500, 2500, 6
    rng = np.random.default_rng(56)

    def lp(long_row):
        rows = np.sort(rng.permuted(np.tile(np.arange(1, m), (n, 1)), axis=1)[:, :per], axis=1)
        if long_row:
            rows[:, 0] = 0
        base = G.random_lp(m, n, 3.0, m // 2, 57)
        return type(base)(num_rows=m, num_cols=n, start=np.arange(n + 1) * per, index=rows.ravel(),
                          value=rng.standard_normal(n * per), col_cost=base.col_cost, col_lower=base.col_lower,
                          col_upper=base.col_upper, row_lower=base.row_lower, row_upper=base.row_upper)

    for long_row in (False, True, False):
        _check([lp(long_row) for _ in range(3)], 0, 130)
