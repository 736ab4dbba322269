"""The pivoted panel kernel with long slabs in shared memory, where update and dot
products of a stage are one pass or two, against LAPACK dgeqp3."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(29100, 30), (29300, 70), (30000, 128), (50000, 41), (40000, 80)])
def test_long_slabs(hq, m, n):
    import scipy.linalg as sl
    A = oracle.gaussian(m, n, m + n)
    hq.set_precision(hq.PLAIN)
    F, jp, tau, info, _ = hq.dgeqp4(A)
    assert info == 0
    (Fo, to), Ro, po = sl.qr(A, mode="raw", pivoting=True)
    np.testing.assert_array_equal(jp, po + 1)
    R, Rr = np.triu(F[:n]), np.triu(Ro[:n])
    assert np.max(np.linalg.norm(R - Rr, axis=0) / np.linalg.norm(Rr, axis=0)) <= 1e-12
    assert np.max(np.abs(np.tril(F, -1) - np.tril(Fo, -1))) <= 1e-12
    assert np.max(np.abs(tau - to)) <= 1e-12
