"""Implied bounds in both forms (grid; one block a case, in shared memory): the same bounds bit for bit.  The grid form
is reached by what is put beside an LP without touching it: columns in no row (the vectors no longer fit a block), or
rows without sides (the operators no longer do; with fewer of those the block form stays, with more threads)."""
import numpy as np
import pytest

import lp_cases
from pramana_b200 import generators as G
from pramana_b200 import pdhg
from pramana_b200 import warmstart as W
from pramana_b200.model import LpCase, Model

pytestmark = pytest.mark.gpu


def _beside(lp, cols, rows, per):
    """lp, `rows` rows without sides over `cols` more columns in [0, 1], `per` entries a column."""
    rng = np.random.default_rng(61)
    at = np.sort(rng.permuted(np.tile(np.arange(rows), (cols, 1)), axis=1)[:, :per], axis=1) + lp.num_rows
    inf = np.full(rows, np.inf)
    return Model(num_rows=lp.num_rows + rows, num_cols=lp.num_cols + cols,
                 start=np.concatenate([lp.start, lp.start[-1] + per * np.arange(1, cols + 1)]),
                 index=np.concatenate([lp.index, at.ravel()]),
                 value=np.concatenate([lp.value, rng.standard_normal(at.size)]),
                 col_cost=np.concatenate([lp.col_cost, np.zeros(cols)]),
                 col_lower=np.concatenate([lp.col_lower, np.zeros(cols)]),
                 col_upper=np.concatenate([lp.col_upper, np.ones(cols)]),
                 row_lower=np.concatenate([lp.row_lower, -inf]), row_upper=np.concatenate([lp.row_upper, inf]))


def _lp(which):
    if which == "refinery":
        return W.RefineryFamily(seed=5, periods=2, regions=1, units=4, streams=4, properties=2, scale_exponent=0.0).base
    if which == "random_free":
        lp = G.random_lp(127, 300, 4.0, 60, 62)
        lp.col_upper[::3] = np.inf
        lp.col_lower[::5] = -np.inf
        return lp
    return lp_cases.edge_lp(7) if which == "edge" else G.random_lp(1, 1, 1.0, 1, 63)


@pytest.mark.parametrize("which", ["refinery", "random_free", "edge", "one"])
@pytest.mark.parametrize("cols,rows,per", [(20000, 1, 0), (1100, 40, 15), (200, 40, 15)])
def test_forms_agree(which, cols, rows, per):
    lp = _lp(which)
    wide = _beside(lp, cols, rows, per)
    rng = np.random.default_rng(64)
    cuts = [rng.uniform(0.5, 1.5, size=lp.num_cols) for _ in range(3)]
    ups = [np.where(np.isfinite(lp.col_upper), np.maximum(lp.col_lower, lp.col_upper * f), lp.col_upper) for f in cuts]
    lo, up = pdhg.impliedBounds(lp, [LpCase()] + [LpCase(col_upper=u) for u in ups])
    wlo, wup = pdhg.impliedBounds(wide, [LpCase()] + [LpCase(col_upper=np.concatenate([u, np.ones(cols)])) for u in ups])
    for b in range(4):
        if np.any(lo[b] > up[b]):
            continue  # crossed before the first round
        assert np.array_equal(lo[b], wlo[b][:lp.num_cols]) and np.array_equal(up[b], wup[b][:lp.num_cols])
