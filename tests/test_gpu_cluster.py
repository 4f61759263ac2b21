"""The resident form on one cluster of 8 blocks: LPs with fewer rows or columns than blocks, with rows on the warp path,
the largest that fit and the first that do not, in both precisions; several prepared LPs at once."""
import numpy as np
import pytest

from oracle import oracle as O
from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G

pytestmark = pytest.mark.gpu


def _blocks(lp, **kw):
    with pdhg.Engine(lp, pdhg.PdhgOptions(**kw)) as eng:
        r = eng.solve()[0]
        return eng.last_stats.resident_blocks, r


# with 5 entries a column 2,400 x 4,800 takes 187 KB of a block in FP64, 3,000 x 6,000 more than the 226 KB there are
@pytest.mark.parametrize("m,n,per,blocks", [(1, 1, 1.0, 8), (3, 2, 2.0, 8), (7, 20, 3.0, 8), (8, 8, 4.0, 8),
                                            (33, 1500, 6.0, 8), (1000, 2000, 5.0, 8), (2000, 4000, 5.0, 8),
                                            (2400, 4800, 5.0, 8), (3000, 6000, 5.0, 148)])
@pytest.mark.parametrize("iters", [1, 64, 193])
def test_iterates(m, n, per, blocks, iters):
    lp = G.random_lp(m, n, min(per, m), m // 2, 17)
    used, r = _blocks(lp, tolerance=1e-30, maxIterations=iters)
    o = O.solve(lp, "oracle", tolerance=1e-30, max_iterations=iters)
    assert used == blocks
    for a, b in ((r.x, o.x), (r.rowDual, o.y)):
        assert np.max(np.abs(a - b)) <= 1e-9 * max(1.0, np.max(np.abs(b)))


@pytest.mark.parametrize("m,n,blocks", [(3, 2, 8), (300, 600, 8), (1500, 3000, 8)])
def test_mixed(m, n, blocks):
    lp = G.random_lp(m, n, min(4.0, m), m // 2, 18)
    used, r = _blocks(lp, tolerance=1e-6, precision=_lib.PRECISION_MIXED)
    o = O.solve(lp, "oracle", tolerance=1e-6)
    assert used == blocks and r.status == "Optimal"
    assert pdhg.kktResidual(lp, r.x, r.rowDual)[0, 3] <= 1e-6 * (1 + 1e-9)
    assert abs(r.objective - o.objective) <= 1e-5 * (1 + abs(o.objective))


def test_prepared_lps_side_by_side():
    """Engines of different shared-memory needs, solved in every order."""
    lps = [G.random_lp(m, 2 * m, 5.0, m // 2, 19) for m in (2000, 50, 6000, 3000)]
    engines = [pdhg.Engine(lp, pdhg.PdhgOptions(tolerance=1e-30, maxIterations=70)) for lp in lps]
    first = [e.solve()[0] for e in engines]
    again = [e.solve()[0] for e in reversed(engines)][::-1]
    for a, b in zip(first, again):
        assert np.array_equal(a.x, b.x) and np.array_equal(a.rowDual, b.rowDual)
    for e in engines:
        e.close()
