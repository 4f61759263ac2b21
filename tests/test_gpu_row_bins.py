"""Row-length bins of the fused kernels on both sides of their rules: operators within and beyond one wave of threads,
with few and with many rows past two rounds of a lane, and rows of 23 to 26 entries (24 is where the wide short path
ends)."""
import numpy as np
import pytest

from oracle import oracle as O
from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G
from pramana_b200.model import Model

pytestmark = pytest.mark.gpu


def _close(lp, r, iters):
    o = O.solve(lp, "oracle", tolerance=1e-30, max_iterations=iters)
    for a, b in ((r.x, o.x), (r.rowDual, o.y)):
        assert np.max(np.abs(a - b)) <= 1e-9 * max(1.0, np.max(np.abs(b)))


@pytest.mark.parametrize("m,n,per", [(30000, 60000, 2.0), (30000, 60000, 6.0), (160000, 200000, 3.0),
                                     (160000, 240000, 8.0)])
def test_random_rows(m, n, per):
    lp = G.random_lp(m, n, per, m // 2, 31)
    po = pdhg.PdhgOptions(tolerance=1e-30, maxIterations=66, kernelMode=_lib.KERNELS_FUSED)
    _close(lp, pdhg.solvePdhg(lp, po), 66)


@pytest.mark.parametrize("rows", [200, 20000])
def test_rows_around_the_short_path(rows):
    """Row i holds 20 + i % 8 entries (and one row 2,100, one row none)."""
    rng = np.random.default_rng(32)
    n = 3000
    lens = 20 + np.arange(rows) % 8
    lens[5], lens[6] = 2100, 0
    row = np.repeat(np.arange(rows), lens)
    col = np.concatenate([rng.choice(n, size=k, replace=False) for k in lens])
    order = np.lexsort((row, col))
    row, col = row[order], col[order]
    start = np.concatenate([[0], np.cumsum(np.bincount(col, minlength=n))])
    val = rng.standard_normal(len(row))
    side = np.bincount(row, val * rng.uniform(0, 1, size=n)[col], minlength=rows)
    lp = Model(num_rows=rows, num_cols=n, start=start, index=row, value=val, col_cost=rng.standard_normal(n),
               col_lower=np.zeros(n), col_upper=np.ones(n), row_lower=np.full(rows, -np.inf), row_upper=side)
    po = pdhg.PdhgOptions(tolerance=1e-30, maxIterations=66, kernelMode=_lib.KERNELS_FUSED)
    _close(lp, pdhg.solvePdhg(lp, po), 66)
    multi = pdhg.solvePdhgMulti([lp, lp], pdhg.PdhgOptions(tolerance=1e-30, maxIterations=66,
                                                           multiForm=_lib.MULTI_GRID))
    for r in multi:
        _close(lp, r, 66)
