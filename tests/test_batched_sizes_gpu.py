"""Batched QR: which matrices the plan gives to teams of CTAs, at the limits of
that rule, and runs whose sizes are not the plan's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _team_counts(bq):
    """How many of the schedule's first matrices go to teams, by CTAs per SM."""
    import torch
    return bq.work[:256].view(torch.int32)[9:16].cpu().tolist()


def _factor(bq, shapes, seed):
    import torch
    As = [oracle.gaussian(m, n, seed + i) for i, (m, n) in enumerate(shapes)]
    mats = [torch.from_numpy(np.ascontiguousarray(A.T)).cuda() for A in As]
    bq.shapes = list(shapes)
    sizes = np.array(shapes, np.int32)
    bq.d_m.copy_(torch.from_numpy(sizes[:, 0].copy()))
    bq.d_n.copy_(torch.from_numpy(sizes[:, 1].copy()))
    bq.d_lda.copy_(torch.from_numpy(sizes[:, 0].copy()))
    jp, tau, info = bq.run(mats)
    torch.cuda.synchronize()
    return As, [t.cpu().numpy().T for t in mats], jp, tau, info.cpu().numpy()


def _check(oracle_lib, As, Fs, jps, taus, info):
    assert not info.any(), [hex(i) for i in info]
    for A, F, jp, tau in zip(As, Fs, jps, taus):
        Ao, jo, to, _ = oracle_lib.dgeqp3(A)
        k, n = min(A.shape), A.shape[1]
        np.testing.assert_array_equal(jp.cpu().numpy()[:n], jo)
        assert np.max(np.abs(tau.cpu().numpy()[:k] - to)) <= TOL
        assert np.max(np.linalg.norm(F - Ao, axis=0) / np.linalg.norm(Ao, axis=0)) <= TOL


# A team's smallest matrix, its most rows and one more, a matrix with fewer
# columns than a team has warps; the counts hold for every number of CTAs per
# SM here, each matrix being a large part of the batch.
@pytest.mark.parametrize("shapes,count", [
    ([(128, 128)], 1), ([(127, 129)], 0), ([(1024, 16)], 1), ([(1023, 16)], 0), ([(1024, 17)], 1),
    ([(1025, 40)], 0), ([(700, 24), (128, 128)], 2), ([(16, 1024)], 1),
    ([(1024, 60), (1025, 40), (128, 128)], 1)])
@pytest.mark.parametrize("cfg", [3, 4, 5, 6])
def test_team_limits(hq, oracle_lib, shapes, count, cfg):
    bq = hq.BatchedQRP(shapes, autotune=False)
    assert _team_counts(bq) == [count] * 7
    bq.cfg = cfg
    _check(oracle_lib, *_factor(bq, shapes, 40))


# Teams of four (shape 4) by default only where a few matrices are long beside
# the rest: alone, or before many small ones; not when as many equal matrices as
# CTAs, or more, keep every CTA at work.
@pytest.mark.parametrize("shapes,cfg", [
    ([(128, 128)], 4), ([(128, 128)] * 304, 1), ([(128, 128)] * 1000, 1), ([(300, 300)] * 20, 4),
    ([(300, 300)] * 304, 1), ([(1000, 500)] + [(40, 30)] * 500, 4), ([(60, 50)] * 10, 1)])
def test_default_shape(hq, shapes, cfg):
    assert hq.BatchedQRP(shapes, autotune=False).cfg == cfg


# Columns on both sides of 1024 rows, where they no longer stay in registers,
# and of the 32 rows that one step of a warp takes; narrow and wide ones.
LONG = [(1024, 40), (1025, 40), (1055, 33), (1056, 1), (1057, 2), (2049, 20), (5000, 3), (1030, 129),
        (31, 7), (32, 33), (33, 200), (1, 5)]


@pytest.mark.parametrize("cfg", range(9))
def test_long_columns(hq, oracle_lib, cfg):
    bq = hq.BatchedQRP(LONG, autotune=False)
    bq.cfg = cfg
    _check(oracle_lib, *_factor(bq, LONG, 100))


@pytest.mark.parametrize("cfg", range(9))
def test_sizes_that_are_not_the_plans(hq, oracle_lib, cfg):
    """Planned for a team with up to 1024 rows, more than that when run; others
    grow, shrink and vanish."""
    plan = [(800, 300), (600, 200), (300, 200), (1500, 60), (20, 10), (40, 300)]
    now = [(1300, 290), (1025, 120), (1024, 200), (700, 60), (200, 150), (1, 1)]
    bq = hq.BatchedQRP(plan, autotune=False)
    assert min(_team_counts(bq)) >= 2
    # Outputs large enough for both.
    import torch
    bq.jpvt = [torch.zeros(300, dtype=torch.int32, device="cuda") for _ in plan]
    bq.tau = [torch.zeros(300, dtype=torch.float64, device="cuda") for _ in plan]
    bq.cfg = cfg
    _check(oracle_lib, *_factor(bq, now, 70))
