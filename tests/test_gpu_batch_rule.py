"""Batches whose kernel variant comes from their size: the same iterates, bit for bit, as the plain variant's, on
both sides of the rule's lines and across a compaction."""
import numpy as np
import pytest

from pramana_b200 import generators as G
from pramana_b200 import pdhg
from pramana_b200.model import LpCase

pytestmark = pytest.mark.gpu


# 3 x 2^19 elements (rows + columns times cases) is where the variant changes: 524,288 columns and rows at 3 cases; row
# tiles from there on for 28..32, 56..64, ... cases
@pytest.mark.parametrize("rows,cases,tol", [(174762, 3, 1e-30), (174763, 3, 1e-30), (18724, 28, 1e-30),
                                            (18725, 28, 1e-30), (19500, 27, 1e-30), (9400, 56, 1e-30),
                                            (8600, 61, 1e-4), (37, 2, 1e-4), (37, 61, 1e-4)])
def test_rule_changes_no_iterate(rows, cases, tol):
    lp = G.random_lp(rows, 2 * rows, 4.0, rows // 2, 8)
    rng = np.random.default_rng(cases)
    cs = [LpCase(cost=lp.col_cost * rng.uniform(0.5, 1.5, size=2 * rows)) for _ in range(cases)]
    po = dict(tolerance=tol, maxIterations=130 if tol < 1e-20 or rows > 1000 else 20000)
    got, plain = [pdhg.solvePdhgBatch(lp, cs, pdhg.PdhgOptions(batchVariant=v, **po)) for v in (0, 1)]
    for a, b in zip(got, plain):
        assert a.iterations == b.iterations and np.array_equal(a.x, b.x) and np.array_equal(a.rowDual, b.rowDual)
