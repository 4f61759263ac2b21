"""Set-up of many LPs on the device (pdhg_members.cuh): members that share one operator get bit for bit what they get
with an operator each, and what the oracle gets before the first check, at the edges of the kernels' blocks (256
elements, 1,024 terms of a sum, two terms a row) and with every kind of bound."""
import numpy as np
import pytest

from oracle import oracle as O
from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G
from pramana_b200.model import Model

pytestmark = pytest.mark.gpu


def _members(m, n, count):
    base = G.random_lp(m, n, min(3.0, m), m // 2, 21)
    rng = np.random.default_rng(22)
    out = []
    for _ in range(count):
        lo, up = base.col_lower.copy(), base.col_upper.copy()
        lo[rng.random(n) < 0.2] = -np.inf
        up[rng.random(n) < 0.2] = np.inf
        up[rng.random(n) < 0.1] = 1e21  # infinite too
        lo[rng.random(n) < 0.1] = 2.0
        rl, ru = base.row_lower.copy(), base.row_upper.copy()
        free = rng.random(m) < 0.1
        rl[free], ru[free] = -np.inf, np.inf
        out.append(Model(num_rows=m, num_cols=n, start=base.start, index=base.index, value=base.value,
                         col_cost=base.col_cost * rng.uniform(0.1, 10.0, size=n), col_lower=lo, col_upper=up,
                         row_lower=rl, row_upper=ru, obj_offset=float(rng.standard_normal())))
    return out


@pytest.mark.parametrize("m,n", [(1, 1), (255, 256), (257, 255), (511, 513), (512, 1023), (513, 1025), (1030, 2049)])
@pytest.mark.parametrize("warm", [False, True])
def test_shared_operator_changes_nothing(m, n, warm):
    lps = _members(m, n, 5)
    other = G.random_lp(m + 1, n + 1, 2.0 if m > 1 else 1.0, 1, 23)  # beside it, every LP has its own operator
    rng = np.random.default_rng(24)
    starts = [(rng.standard_normal(n), rng.standard_normal(m)) for _ in lps] if warm else None
    weights = rng.uniform(0.5, 2.0, size=5) if warm else None
    for iters in (3, 130):
        po = pdhg.PdhgOptions(tolerance=1e-30, maxIterations=iters, multiForm=_lib.MULTI_CTA,
                              ctaThreads=256, ctaKernel=_lib.CTA_GENERAL)  # one variant: its check sums have one order
        one = pdhg.solvePdhgMulti(lps, po, starts=starts, primalWeights=weights)
        each = pdhg.solvePdhgMulti(lps + [other], po, starts=None if starts is None else starts + [None],
                                   primalWeights=None if weights is None else np.append(weights, 0.0))
        for lp, a, b in zip(lps, one, each):
            assert np.array_equal(a.x, b.x) and np.array_equal(a.rowDual, b.rowDual)
            assert (a.objective, a.relativeKkt, a.primalWeight) == (b.objective, b.relativeKkt, b.primalWeight)
            if iters == 3 and not warm:
                o = O.solve(lp, "oracle", tolerance=1e-30, max_iterations=3)
                assert np.array_equal(a.x, o.x) and np.array_equal(a.rowDual, o.y)


@pytest.mark.parametrize("form", [_lib.MULTI_GRID, _lib.MULTI_CTA])
def test_degenerate_members(form):
    """One LP alone, LPs without rows, without entries, and members over equal (not the same) arrays."""
    po = pdhg.PdhgOptions(tolerance=1e-6, maxIterations=500, multiForm=form)
    empty = Model(num_rows=0, num_cols=3, start=np.zeros(4), index=np.zeros(0), value=np.zeros(0),
                  col_cost=np.array([1.0, -1.0, 0.0]), col_lower=np.zeros(3), col_upper=np.ones(3),
                  row_lower=np.zeros(0), row_upper=np.zeros(0))
    lp = G.random_lp(30, 50, 3.0, 10, 25)
    twin = Model(**{f: (np.copy(getattr(lp, f)) if isinstance(getattr(lp, f), np.ndarray) else getattr(lp, f))
                    for f in ("num_rows", "num_cols", "start", "index", "value", "col_cost", "col_lower", "col_upper",
                              "row_lower", "row_upper", "obj_offset")})
    alone = pdhg.solvePdhgMulti([lp], po)[0]
    for r in pdhg.solvePdhgMulti([lp, twin], po):
        assert np.array_equal(r.x, alone.x) and r.iterations == alone.iterations
    r = pdhg.solvePdhgMulti([empty, empty, lp], po)
    assert np.array_equal(r[0].x, r[1].x) and abs(r[0].objective + 1.0) <= 1e-6
    assert np.max(np.abs(r[2].x - alone.x)) <= 1e-9 * max(1.0, np.max(np.abs(alone.x)))


def test_more_elements_than_the_grid_has_threads():
    """One LP of 65,535 blocks of 256 columns and 300 more, few of them in its three rows."""
    m, n, used = 3, 65535 * 256 + 300, 8
    rng = np.random.default_rng(26)
    at = np.r_[0:used // 2, n - used // 2:n]  # both ends
    counts = np.zeros(n, dtype=np.int64)
    counts[at] = 1
    lp = Model(num_rows=m, num_cols=n, start=np.concatenate([[0], np.cumsum(counts)]), index=np.arange(used) % m,
               value=rng.uniform(1.0, 2.0, size=used), col_cost=rng.standard_normal(n), col_lower=np.zeros(n),
               col_upper=np.ones(n), row_lower=np.full(m, 0.5), row_upper=np.full(m, np.inf))
    po = pdhg.PdhgOptions(tolerance=1e-30, maxIterations=3, multiForm=_lib.MULTI_GRID)
    got = pdhg.solvePdhgMulti([lp], po)[0]
    want = O.solve(lp, "oracle", tolerance=1e-30, max_iterations=3)
    # three steps of separately rounded arithmetic over sums of at most three terms
    assert np.max(np.abs(got.x - want.x)) <= 1e-12 and np.max(np.abs(got.rowDual - want.y)) <= 1e-12
