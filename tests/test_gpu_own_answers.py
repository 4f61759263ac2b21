"""Every answer has memory of its own: what one case's or LP's result keeps is that answer and not the batch's, and
writing to it changes no other; the arrays are those b2p_engine_fetch gives, around the halves the copies go through."""
import ctypes as C

import numpy as np
import pytest

from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G
from pramana_b200.model import LpCase

pytestmark = pytest.mark.gpu


def _own(results):
    for r in results:
        for a in (r.x, r.rowDual):
            assert a.base is None and a.flags.owndata and a.flags.writeable and a.dtype == np.float64


def _cases(lp, k):
    rng = np.random.default_rng(91)
    return [LpCase(cost=lp.col_cost * rng.uniform(0.9, 1.1, lp.num_cols)) for _ in range(k)]


# the halves hold 2^18 doubles: one case and many in a half, a case over several, a half that ends with a case
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 5, 2), (40, 70, 9), (1024, 1 << 14, 33), (1 << 15, 1 << 15, 17),
                                   (300, 300_001, 2), (300, 1 << 18, 3), (20, 600_000, 1)])
def test_batch(m, n, k):
    lp = G.random_lp(m, n, 1.0, m // 2, 92)
    opts = pdhg.PdhgOptions(tolerance=1e-30, maxIterations=40, useGraphs=False)
    cases = _cases(lp, k)
    with pdhg.Engine(lp, opts, cases) as e:
        got = e.solve()
        x, y = e.fetch()
    _own(got)
    for b, r in enumerate(got):
        assert np.array_equal(r.x, x[b * n:(b + 1) * n]) and np.array_equal(r.rowDual, y[b * m:(b + 1) * m])
    assert len({r.x.ctypes.data for r in got}) == k
    called = pdhg.solvePdhgBatch(lp, cases, opts)
    _own(called)
    for a, b in zip(called, got):
        assert np.array_equal(a.x, b.x) and np.array_equal(a.rowDual, b.rowDual) and a.objective == b.objective
    got[0].x[:] = 7.0
    assert k == 1 or np.array_equal(got[1].x, called[1].x)


@pytest.mark.parametrize("form", [_lib.MULTI_GRID, _lib.MULTI_CTA])
def test_many(form):
    lps = [G.random_lp(m, n, 2.0, m // 2, 93 + m) for m, n in ((1, 1), (5, 9), (300, 200), (40, 70))]
    got = pdhg.solvePdhgMulti(lps, pdhg.PdhgOptions(tolerance=1e-30, maxIterations=40, multiForm=form))
    _own(got)
    assert [(len(r.x), len(r.rowDual)) for r in got] == [(lp.num_cols, lp.num_rows) for lp in lps]
    one = pdhg.solvePdhg(lps[2], pdhg.PdhgOptions(tolerance=1e-30, maxIterations=40))
    _own([one])
    np.testing.assert_allclose(got[2].x, one.x, rtol=1e-9, atol=1e-12)


def test_left_out_entries():
    lp = G.random_lp(30, 50, 3.0, 9, 94)
    with pdhg.Engine(lp, pdhg.PdhgOptions(tolerance=1e-30, maxIterations=40), _cases(lp, 3)) as e:
        want = e.solve()
        x = [np.full(lp.num_cols, -1.0) for _ in range(3)]
        px = (_lib.dptr * 3)(x[0].ctypes.data_as(_lib.dptr), None, x[2].ctypes.data_as(_lib.dptr))
        _lib.check(e._lib.b2p_engine_fetch_cases(e._h, px, None))
        assert np.array_equal(x[0], want[0].x) and (x[1] == -1.0).all() and np.array_equal(x[2], want[2].x)
        assert e._lib.b2p_engine_fetch_cases(e._h, None, None) == 0
    with pdhg.Engine(lp, pdhg.PdhgOptions(), _cases(lp, 3)) as e:  # nothing solved: nothing written
        x[1][:] = 5.0
        px[1] = x[1].ctypes.data_as(_lib.dptr)
        _lib.check(e._lib.b2p_engine_fetch_cases(e._h, px, None))
        assert (x[1] == 5.0).all()
    assert e._lib.b2p_engine_fetch_cases(C.c_void_p(), None, None) == 1
