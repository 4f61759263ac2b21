"""Sums in a fixed serial order (csrc/pdhg_ordered.cuh) at the edges of their chunks of 1,024 terms: the certified
bound against the same additions in exact rational arithmetic, the spectral norms of many LPs through iterates that
equal the oracle's bit for bit."""
import math
from fractions import Fraction

import numpy as np
import pytest

from oracle import oracle as O
from pramana_b200 import generators as G
from pramana_b200 import _lib, pdhg
from pramana_b200.model import Model

pytestmark = pytest.mark.gpu


def _add_down(a, b):
    s = a + b
    if not math.isfinite(s):
        return s
    return math.nextafter(s, -math.inf) if Fraction(a) + Fraction(b) < Fraction(s) else s


@pytest.mark.parametrize("rows", [1, 2, 1022, 1023, 1024, 1025, 2048, 2049, 5000])
@pytest.mark.parametrize("kind", ["mixed", "cancel", "overflow"])
def test_bound_is_the_downward_sum_in_order(rows, kind):
    """No entries, y = scale: the terms are scale * b_i exactly (a power of two) and the columns' are zero."""
    rng = np.random.default_rng(rows)
    b = rng.standard_normal(rows) * 10.0 ** rng.uniform(-12, 12, size=rows)
    scale = 1.0
    if kind == "cancel":
        b[1::2] = -b[:rows - 1:2][:len(b[1::2])]
    elif kind == "overflow":
        b, scale = rng.choice([-1.0, 1.0], size=rows) * 1e19, 2.0 ** 960
    lp = Model(num_rows=rows, num_cols=2, start=np.zeros(3), index=np.zeros(0), value=np.zeros(0),
               col_cost=np.zeros(2), col_lower=np.zeros(2), col_upper=np.ones(2), row_lower=b, row_upper=b)
    want = 0.0
    for v in b * scale:
        want = _add_down(want, float(v))
    got = pdhg.safeDualBound(lp, np.full(rows, scale))[0]["bound"]
    assert got == want and math.copysign(1.0, got) == math.copysign(1.0, want)


def test_norms_of_many_lps_bit_identical():
    """Column counts on both sides of one and two chunks: the steps of every LP come from its norm, so iterates
    that equal the oracle's bit for bit pin the norms."""
    lps = [G.random_lp(60, n, 3.0, 30, seed) for seed, n in enumerate((1, 31, 1023, 1024, 1025, 2048, 2049))]
    res = pdhg.solvePdhgMulti(lps, pdhg.PdhgOptions(tolerance=1e-30, maxIterations=3,
                                                    multiForm=_lib.MULTI_CTA))
    for lp, r in zip(lps, res):
        o = O.solve(lp, "oracle", tolerance=1e-30, max_iterations=3)
        assert np.array_equal(r.x, o.x) and np.array_equal(r.rowDual, o.y)
