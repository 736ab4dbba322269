"""Split products of K <= 256 (their 64-bit sums): digits at their largest,
tile and K-block remainders, several tiles a CTA, every digit count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _col(X):
    import torch
    return torch.from_numpy(np.ascontiguousarray(X.T)).cuda()


def _bound(s):
    """Relative to |A| |B| for entries of [1/2, 1) times their row's scale
    (hence the 4): s + 3 digit pairs and remainders of 2^-8s each are dropped;
    the level-4 accumulator takes 5 K/16 rounded additions of integers up to
    2^25 in units of 2^-46 (at most 2 each over K = 256: 2^-45), and the FP64
    reference sums K terms (2^-45)."""
    return 4 * (s + 3) * 2.0 ** (-8 * s) + 4 * 2.0 ** -44


@pytest.mark.parametrize("m,n,k,s", [
    (1, 1, 1, 7), (127, 79, 31, 7), (129, 81, 33, 7), (128, 80, 32, 7), (130, 161, 255, 7),
    (257, 240, 256, 7), (5120, 641, 256, 7), (300, 90, 256, 6), (129, 81, 64, 5),
    (129, 81, 256, 4), (60, 90, 100, 3), (60, 90, 256, 2), (129, 81, 256, 1),
])
@pytest.mark.parametrize("kind", ["same sign", "all digits -128", "random"])
def test_short_products(hq, m, n, k, s, kind):
    rng = np.random.default_rng(m + n + k + s)
    if kind == "same sign":      # top digit 128: the largest sums
        A, B = np.full((m, k), 1 - 2.0 ** -53), np.full((k, n), 1 - 2.0 ** -53)
    elif kind == "all digits -128":  # -(127/128 + 128/2^15 + 128/2^23 + ...)
        x = -(127 / 128 + sum(128.0 * 2.0 ** (-7 - 8 * i) for i in range(1, 6)))
        A, B = np.full((m, k), x), np.full((k, n), x)
    else:
        A, B = rng.uniform(0.5, 1, (m, k)), rng.uniform(0.5, 1, (k, n))
        A *= rng.choice([-1.0, 1.0], A.shape)
    A = A * 2.0 ** rng.integers(-300, 300, (m, 1))
    B = B * 2.0 ** rng.integers(-300, 300, (1, n))
    C0 = rng.standard_normal((m, n)) * (np.abs(A) @ np.abs(B))
    for beta, sign in ((0.0, 1.0), (1.0, -1.0)):
        C = _col(C0)
        hq.ozaki_dgemm("N", "N", sign, _col(A), _col(B), beta, C, slices=s)
        err = np.abs(C.cpu().numpy().T - (beta * C0 + sign * (A @ B)))
        # The update's FP64 addition adds half a unit in the last place of the
        # sum, at most 8 times |A| |B| here.
        assert (err / (np.abs(A) @ np.abs(B))).max() <= _bound(s) + beta * 8 * 2.0 ** -53


def test_short_product_zero_and_range_limits(hq):
    A = np.zeros((3, 4))
    A[1] = 2.0 ** -600
    A[2] = -2.0 ** 500
    B = np.full((4, 2), 2.0 ** -600)
    B[:, 1] = 2.0 ** 500
    import torch
    C = torch.full((2, 3), 7.0, dtype=torch.float64, device="cuda")
    hq.ozaki_dgemm("N", "N", 1.0, _col(A), _col(B), 0.0, C, slices=7)
    got = C.cpu().numpy().T
    # Below the normal range: zero.
    np.testing.assert_array_equal(got, [[0, 0], [0, 2.0 ** -98], [-2.0 ** -98, -2.0 ** 1002]])
    assert not np.signbit(got[0]).any() and not np.signbit(got[1, 0])
