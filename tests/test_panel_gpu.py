"""The pivoted panel kernel over its launch shapes and rare paths, through
dgeqp4's small-matrix branch, against LAPACK dgeqp3 on the same matrix:
columns at the limits of its shapes (128 / 129, 512 / 513, 1024), slabs of one
row to slabs that do not fit shared memory, norm recomputations, non-finite
input."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _check(hq, A, tol=1e-12):
    import scipy.linalg as sl
    m, n = A.shape
    k = min(m, n)
    hq.set_precision(hq.PLAIN)
    F, jp, tau, info, _ = hq.dgeqp4(A)
    assert info == 0
    (Fo, to), Ro, po = sl.qr(A, mode="raw", pivoting=True)
    np.testing.assert_array_equal(jp, po + 1)
    R, Rr = np.triu(F[:k]), np.triu(Ro[:k])
    assert np.max(np.linalg.norm(R - Rr, axis=0) / np.linalg.norm(Rr, axis=0)) <= tol
    V, Vo = np.tril(F[:, :k], -1), np.tril(Fo[:, :k], -1)
    assert np.max(np.abs(V - Vo)) <= tol * max(1.0, np.max(np.abs(Vo)))
    assert np.max(np.abs(tau - to)) <= tol


@pytest.mark.parametrize("m,n", [
    (1, 1), (2, 7), (17, 16), (300, 127), (300, 128), (300, 129), (700, 512), (700, 513),
    (520, 1024), (999, 998), (5000, 64), (3001, 260), (30000, 150)])
def test_shapes(hq, m, n):
    _check(hq, oracle.gaussian(m, n, 3 * m + n))


@pytest.mark.parametrize("m,n", [(400, 100), (400, 300), (25000, 140)])
def test_recomputed_norms(hq, m, n):
    """Columns close to the span of a few leading ones: their norms cancel and
    are recomputed, several columns in one stage; the last size works in place
    in global memory."""
    rng = np.random.default_rng(m + n)
    B = rng.standard_normal((m, 5))
    scale = 10.0 ** -rng.uniform(5.0, 6.0, n)
    A = np.asfortranarray(B @ rng.standard_normal((5, n)) + rng.standard_normal((m, n)) * scale)
    import scipy.linalg as sl
    hq.set_precision(hq.PLAIN)
    F, jp, tau, info, _ = hq.dgeqp4(A)
    assert info == 0 and sorted(jp) == list(range(1, n + 1))
    Ro, po = sl.qr(A, mode="r", pivoting=True)[:2]
    np.testing.assert_array_equal(jp, po + 1)
    d, do = np.abs(np.diag(F)[:n]), np.abs(np.diag(Ro))
    # Backward stable: R's diagonal is off by a few eps of the matrix.
    assert np.max(np.abs(d - do)) <= 50.0 * n * np.finfo(float).eps * do[0]


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("m,n", [(96, 64), (300, 200)])
def test_non_finite_input_ends(hq, m, n, bad):
    """Non-finite entries give non-finite results, not an error status or a
    wait that runs out, and a valid permutation."""
    A = oracle.gaussian(m, n, 9)
    A[m // 2, n // 3] = bad
    hq.set_precision(hq.PLAIN)
    F, jp, tau, info, _ = hq.dgeqp4(A)
    assert info == 0 and sorted(jp) == list(range(1, n + 1))
    assert not np.all(np.isfinite(F))


# The column-partitioned kernel (more than 512 columns, at most 1024 rows): one
# and several columns a CTA, columns in registers four, two and one at a time,
# a matrix that does not fit the grid's shared memory, one row.
@pytest.mark.parametrize("m,n", [
    (1, 600), (7, 513), (40, 1100), (129, 700), (257, 2000), (513, 900), (1000, 999), (999, 5200)])
def test_wide_shapes(hq, m, n):
    _check(hq, oracle.gaussian(m, n, 5 * m + n))


def test_wide_recomputed_norms(hq):
    import scipy.linalg as sl
    rng = np.random.default_rng(8)
    m, n = 300, 1500
    A = np.asfortranarray(rng.standard_normal((m, 5)) @ rng.standard_normal((5, n))
                          + rng.standard_normal((m, n)) * 10.0 ** -rng.uniform(5.0, 6.0, n))
    hq.set_precision(hq.PLAIN)
    F, jp, tau, info, _ = hq.dgeqp4(A)
    Ro, po = sl.qr(A, mode="r", pivoting=True)[:2]
    np.testing.assert_array_equal(jp, po + 1)
    d, do = np.abs(np.diag(F)), np.abs(np.diag(Ro))
    assert np.max(np.abs(d - do)) <= 50.0 * m * np.finfo(float).eps * do[0]


def test_wide_wait_that_gives_up(hq):
    A = oracle.gaussian(200, 1200, 4)
    hq.set_precision(hq.PLAIN)
    want = hq.dgeqp4(A)
    hq.set_spin_limit(1)
    try:
        with pytest.raises(hq.HQRRPError, match="barrier"):
            hq.dgeqp4(A)
    finally:
        hq.set_spin_limit(0)
    for w, g in zip(want[:3], hq.dgeqp4(A)[:3]):
        np.testing.assert_array_equal(w, g)
