"""The CTA form's remembered kernel choice: a batch of LPs with operators of their own does not inherit the one timed on
a batch of the same sizes that shares its operator, nor the other way about; each kind is timed once."""
import numpy as np
import pytest

from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.PRECISION_FP64, _lib.PRECISION_MIXED])
@pytest.mark.parametrize("shared_first", [False, True])
def test_shared_and_own_operators_are_timed_apart(shared_first, precision):
    # sizes no other test uses: the choice lives as long as the process
    m, n = 407 + shared_first, 611 + 2 * precision
    base = G.random_lp(m, n, 4.0, 150, 81)

    def member(i, own):
        value = np.array(base.value)
        value[0] += 0.25 * i * own
        return type(base)(num_rows=m, num_cols=n, start=base.start, index=base.index, value=value,
                          col_cost=base.col_cost, col_lower=base.col_lower, col_upper=base.col_upper,
                          row_lower=base.row_lower, row_upper=base.row_upper)

    def tuned(own):
        pdhg.solvePdhgMulti([member(i, own) for i in range(3)],
                            pdhg.PdhgOptions(tolerance=1e-30, maxIterations=400, precision=precision,
                                             multiForm=_lib.MULTI_CTA))
        return pdhg.solvePdhgMulti.last_stats.autotune_seconds > 0

    own_first = not shared_first
    assert [tuned(own_first), tuned(not own_first), tuned(own_first), tuned(not own_first)] == [True, True, False, False]
