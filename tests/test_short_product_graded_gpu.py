"""Split products of K <= 256 whose results are small beside their row's and
column's scales: every bit of the seven digits counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _col(X):
    import torch
    return torch.from_numpy(np.ascontiguousarray(X.T)).cuda()


@pytest.mark.parametrize("m,n,k", [(1, 3, 2), (5, 81, 4), (129, 80, 31), (128, 161, 64), (300, 90, 128),
                                   (257, 240, 256)])
def test_single_entries_come_through(hq, m, n, k):
    """Rows with one entry, a power of two, pick entries of B that are graded
    over all of the digits' 54 bits below their column's largest: each product
    of digits is exact, none is dropped, and so is the result."""
    rng = np.random.default_rng(m + n + k)
    pick = rng.integers(0, k, m)
    A = np.zeros((m, k))
    A[np.arange(m), pick] = rng.choice([-1.0, 1.0], m) * 2.0 ** rng.integers(-200, 200, m)
    bits = rng.integers(1, 54, (k, n))
    B = np.floor(rng.uniform(0.5, 1, (k, n)) * 2.0 ** bits) * 2.0 ** -54
    B *= rng.choice([-1.0, 1.0], B.shape)
    B[rng.integers(0, k, n), np.arange(n)] = 1.0
    B *= 2.0 ** rng.integers(-200, 200, n)
    want = A[np.arange(m), pick][:, None] * B[pick]
    for beta in (0.0, 1.0):
        C = _col(np.zeros((m, n)))
        hq.ozaki_dgemm("N", "N", 1.0, _col(A), _col(B), beta, C, slices=7)
        np.testing.assert_array_equal(C.cpu().numpy().T, want)
