"""Answers out of the k-interleaved scaled space (k_answers) at the edges of its 32 x 32 tiles: every case of a batch
gets bit for bit what it gets beside a copy of itself, whether the cases end together or check by check."""
import numpy as np
import pytest

from pramana_b200 import generators as G
from pramana_b200 import pdhg
from pramana_b200.model import LpCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cases", [2, 31, 32, 33, 65])
@pytest.mark.parametrize("rows,cols", [(1, 2), (31, 33), (64, 96)])
@pytest.mark.parametrize("tol", [1e-30, 1e-4])
def test_case_alone_and_in_a_batch(cases, rows, cols, tol):
    lp = G.random_lp(rows, cols, min(3.0, rows), rows // 2, 5)
    rng = np.random.default_rng(cases)
    cs = [LpCase(cost=lp.col_cost * rng.uniform(0.5, 1.5, size=cols)) for _ in range(cases)]
    po = pdhg.PdhgOptions(tolerance=tol, maxIterations=200 if tol < 1e-20 else 20000)
    got = pdhg.solvePdhgBatch(lp, cs, po)
    assert tol < 1e-20 or rows == 1 or len({r.iterations for r in got}) > 1 or cases == 2
    for b in sorted({0, 1, 30, 31, 32, cases - 2, cases - 1} & set(range(cases))):
        one = pdhg.solvePdhgBatch(lp, [cs[b], cs[b]], po)[1]
        assert one.iterations == got[b].iterations and one.status == got[b].status
        assert np.array_equal(one.x, got[b].x) and np.array_equal(one.rowDual, got[b].rowDual)


def test_engine_answers_stay_until_the_next_solve():
    lp = G.random_lp(40, 70, 4.0, 20, 6)
    with pdhg.Engine(lp, pdhg.PdhgOptions(tolerance=1e-30, maxIterations=64)) as eng:
        assert not eng.fetch()[0].any()
        first = eng.solve()[0]
        eng.set_start(np.ones(70), np.ones(40))
        x, y = eng.fetch()
        assert np.array_equal(x, first.x) and np.array_equal(y, first.rowDual)
        assert not np.array_equal(eng.solve()[0].x, first.x)
