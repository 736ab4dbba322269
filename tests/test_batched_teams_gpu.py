"""Batched QR with teams of CTAs: matrices on both sides of every limit of the
team path, staged and in place, against LAPACK dgeqp3; every team size; a
batch whose first queue is everything, and one whose first queue is empty."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _run(hq, shapes, seed, cfg=None):
    import torch
    rng = np.random.default_rng(seed)
    As = [oracle.gaussian(m, n, int(rng.integers(1 << 30))) for m, n in shapes]
    bq = hq.BatchedQRP(shapes, autotune=False)
    if cfg is not None:
        bq.cfg = cfg
    mats = [torch.from_numpy(np.ascontiguousarray(A.T)).cuda() for A in As]
    jp, tau, info = bq.run(mats)
    torch.cuda.synchronize()
    assert int(info.abs().sum()) == 0
    return As, [t.cpu().numpy().T for t in mats], [j.cpu().numpy() for j in jp], \
        [t.cpu().numpy() for t in tau]


def _check(oracle_lib, As, Fs, jps, taus):
    for A, F, jp, tau in zip(As, Fs, jps, taus):
        Ao, jo, to, _ = oracle_lib.dgeqp3(A)
        k = min(A.shape)
        np.testing.assert_array_equal(jp, jo)
        assert np.max(np.abs(tau[:k] - to) / np.maximum(np.abs(to), 1e-300)) <= TOL
        den = np.linalg.norm(Ao, axis=0)
        den[den == 0] = 1
        assert np.max(np.linalg.norm(F - Ao, axis=0) / den) <= TOL


# Few matrices, so every one that may goes to a team: the smallest a team
# takes (128 x 128) and one below, its most rows (1024) and one more, columns
# fewer than a team's warps, one row more and less than columns, matrices that
# fit a team's shared memory and that do not.
TEAM = [(128, 128), (127, 128), (1024, 17), (1025, 40), (1024, 301), (700, 23), (300, 301),
        (301, 300), (257, 129), (513, 33), (1000, 512), (90, 400)]


@pytest.mark.parametrize("cfg", range(7))
def test_teams_match_lapack(hq, oracle_lib, cfg):
    _check(oracle_lib, *_run(hq, TEAM, 1, cfg))


@pytest.mark.parametrize("shapes", [
    [(200, 150)], [(33, 9)] * 40, [(640, 400), (20, 10), (1, 1), (30, 60)] * 5])
def test_default_shape(hq, oracle_lib, shapes):
    _check(oracle_lib, *_run(hq, shapes, 2))


def test_recomputed_norms_and_non_finite(hq):
    """Nearly dependent columns (norm recomputations) give LAPACK's pivots;
    a NaN gives non-finite results and a valid permutation."""
    import scipy.linalg as sl
    import torch
    rng = np.random.default_rng(3)
    shapes = [(400, 120), (900, 300), (60, 40), (500, 200)]
    As = []
    for m, n in shapes:
        B = rng.standard_normal((m, 4)) @ rng.standard_normal((4, n))
        As.append(np.asfortranarray(B + rng.standard_normal((m, n)) * 10.0 ** -rng.uniform(5, 6, n)))
    As[3][100, 50] = np.nan
    bq = hq.BatchedQRP(shapes, autotune=False)
    mats = [torch.from_numpy(np.ascontiguousarray(A.T)).cuda() for A in As]
    jp, tau, info = bq.run(mats)
    torch.cuda.synchronize()
    assert int(info.abs().sum()) == 0
    for i in range(3):
        Ro, po = sl.qr(As[i], mode="r", pivoting=True)[:2]
        np.testing.assert_array_equal(jp[i].cpu().numpy(), po + 1)
        d, do = np.abs(np.diag(mats[i].cpu().numpy().T)), np.abs(np.diag(Ro))
        n = shapes[i][1]
        assert np.max(np.abs(d[:n] - do[:n])) <= 50.0 * n * np.finfo(float).eps * do[0]
    assert sorted(jp[3].cpu().numpy()) == list(range(1, 201))
    assert not np.all(np.isfinite(mats[3].cpu().numpy()))
