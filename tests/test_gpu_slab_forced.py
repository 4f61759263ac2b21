"""The slab kernel asked for by name, so that what ran is known: every cluster size, both variants, both precisions, at
the edges of a slice (32), of a round of the warps and of a block's shared memory, against the general kernel bit for
bit; and what does not fit is an error."""
import numpy as np
import pytest

from pramana_b200 import _lib, pdhg
from pramana_b200 import generators as G
from pramana_b200 import warmstart as W

pytestmark = pytest.mark.gpu

SLICES = {_lib.CTA_SLAB2: (2, 1), _lib.CTA_SLAB4: (4, 2)}  # of columns, of rows per warp
PRECISIONS = [_lib.PRECISION_FP64, _lib.PRECISION_MIXED]


def _cluster(lps, kernel, size):
    """Blocks of the smallest cluster whose 16 warps and 227 KB a block (less 4 KB of static data) hold every LP: its vectors whole,
    its operators' slices of 32 rows, longest first and dealt out in turn, as wide as their longest row."""
    rc, rr = SLICES[kernel]
    for c in (1, 2, 4, 8):
        fits = True
        for lp in lps:
            m, n = lp.num_rows, lp.num_cols
            entries = sum(32 * int(np.sort(length)[::-1][::32][::c].sum())
                          for length in (np.diff(lp.start), np.bincount(lp.index, minlength=m)))
            need = -(-size * (n + m) // 8) * 8 + -(-size * entries // 8) * 8 + 2 * entries
            fits &= -(-n // (32 * c)) <= 16 * rc and -(-m // (32 * c)) <= 16 * rr and need <= 232448 - 4096
        if fits:
            return c
    return 0


def _run(lps, kernel, iters, tol, precision, threads=0, starts=None):
    return pdhg.solvePdhgMulti(lps, pdhg.PdhgOptions(tolerance=tol, maxIterations=iters, precision=precision,
                                                     multiForm=_lib.MULTI_CTA, ctaKernel=kernel, ctaThreads=threads),
                               starts=starts)


def _check(lps, kernel, iters, tol=1e-30, precision=_lib.PRECISION_FP64, starts=None):
    got = _run(lps, kernel, iters, tol, precision, starts=starts)
    st = pdhg.solvePdhgMulti.last_stats
    mixed = precision == _lib.PRECISION_MIXED
    assert st.cta_cluster == _cluster(lps, kernel, 8) > 0
    assert st.cta_cluster32 == (_cluster(lps, kernel, 4) if mixed else 0)
    assert (st.cta_threads, st.cta_owned_per_thread) == (512, SLICES[kernel][0])
    cluster = st.cta_cluster
    want = _run(lps, _lib.CTA_GENERAL, iters, tol, precision, threads=256, starts=starts)
    st = pdhg.solvePdhgMulti.last_stats
    assert (st.cta_cluster, st.cta_cluster32) == (0, 0)
    for a, b in zip(got, want):
        assert np.array_equal(a.x, b.x) and np.array_equal(a.rowDual, b.rowDual)
        assert (a.status, a.iterations, a.objective, a.relativeKkt) == (b.status, b.iterations, b.objective,
                                                                        b.relativeKkt)
    return cluster


# a cluster of C blocks holds 1,024 C columns and 512 C rows (SLAB2) or 2,048 C and 1,024 C (SLAB4)
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("m,n,per,two,four", [
    (1, 1, 1.0, 1, 1), (31, 33, 3.0, 1, 1), (32, 32, 3.0, 1, 1), (33, 1024, 3.0, 1, 1), (33, 1025, 3.0, 2, 1),
    (500, 2048, 2.0, 2, 1), (500, 2049, 2.0, 4, 2), (512, 900, 3.0, 1, 1), (513, 900, 3.0, 2, 1),
    (1024, 900, 3.0, 2, 1), (1025, 900, 3.0, 4, 2), (1700, 3585, 4.0, 4, 2), (2049, 2000, 8.0, 8, 4),
    (4096, 8192, 1.5, 8, 4)])
@pytest.mark.parametrize("kernel", [_lib.CTA_SLAB2, _lib.CTA_SLAB4])
def test_own_operators(m, n, per, two, four, kernel, precision):
    lps = [G.random_lp(m, n, min(per, m), m // 2, 61 + i) for i in range(2)]
    lps.append(G.random_lp(min(m, 20), min(n, 30), 1.0, min(m, 20) // 2, 60))
    assert _check(lps, kernel, 150, precision=precision) == (two if kernel == _lib.CTA_SLAB2 else four)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("m,n", [(4097, 3000), (8192, 9000)])
def test_eight_blocks_of_four_slices(m, n, precision):
    assert _check([G.random_lp(m, n, 1.5, m // 2, 62)], _lib.CTA_SLAB4, 150, precision=precision) == 8


@pytest.mark.parametrize("precision", PRECISIONS)
def test_bound_by_shared_memory(precision):
    """Few rows and columns, many entries: two blocks in FP64, one in FP32."""
    assert _check([G.random_lp(600, 900, 13.0, 300, 63)], _lib.CTA_SLAB4, 150, precision=precision) == 2


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("kernel", [_lib.CTA_SLAB2, _lib.CTA_SLAB4])
def test_one_operator_to_tolerance(kernel, precision):
    fam = W.RefineryFamily(seed=5, periods=6, regions=2, units=6, streams=6, properties=3, pools=12,
                           scale_exponent=0.0)
    lps = [fam.instance(p) for p in fam.sample(3, seed=64)]
    rng = np.random.default_rng(65)
    starts = [(rng.uniform(0, 10, size=lps[0].num_cols), rng.standard_normal(lps[0].num_rows)), None, None]
    _check(lps, kernel, 3000, tol=1e-3, precision=precision, starts=starts)


def test_more_clusters_than_run_at_once():
    _check([G.random_lp(1025, 900, 3.0, 500, 66 + i % 3) for i in range(200)], _lib.CTA_SLAB4, 100)


@pytest.mark.parametrize("kernel,m,n,threads", [
    (_lib.CTA_SLAB2, 4097, 50, 0), (_lib.CTA_SLAB4, 8193, 50, 0), (_lib.CTA_SLAB2, 50, 8193, 0),
    (_lib.CTA_SLAB4, 50, 16385, 0), (_lib.CTA_SLAB2, 500, 500, 128), (_lib.CTA_SLAB4, 500, 500, 256)])
@pytest.mark.parametrize("precision", PRECISIONS)
def test_refused(kernel, m, n, threads, precision):
    with pytest.raises(_lib.B2pError, match="no CTA kernel variant fits"):
        _run([G.random_lp(m, n, 3.0, 9, 67)], kernel, 100, 1e-6, precision, threads=threads)


def test_unknown_kernel():
    with pytest.raises(_lib.B2pError, match="unknown cta_kernel"):
        _run([G.random_lp(5, 5, 2.0, 2, 68)], _lib.CTA_SLAB4 + 1, 100, 1e-6, _lib.PRECISION_FP64)
