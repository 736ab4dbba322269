"""Pivot selection's launch shapes: one CTA to many clusters, lanes per column
by precision and rows, columns at the edges of what a CTA holds.

Plain runs are compared with the oracle on the same sketch (identical pivots,
tau and R to 1e-12); mixed runs of one matrix embedded in launches of different
shapes must give the same pivots, since a column's arithmetic does not depend
on how columns are laid out.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _plain(hq, oracle_lib, m, n, nb, pp, seed):
    A = oracle.gaussian(m, n, seed)
    G = oracle_lib.sketch(nb + pp, m)
    Ao, jo, to = oracle_lib.hqrrp_sketch(A, G, nb, pp, 1)
    hq.set_precision(hq.PLAIN)
    Ag, jg, tg = hq.hqrrp(A, nb, pp, 1, G=G)
    np.testing.assert_array_equal(jg, jo)
    k = min(m, n)
    R, Ro = np.triu(Ag[:k]), np.triu(Ao[:k])
    assert np.max(np.linalg.norm(R - Ro, axis=0) / np.linalg.norm(Ro, axis=0)) <= 1e-12
    assert np.max(np.abs(tg - to) / np.maximum(np.abs(to), 1e-300)) <= 1e-12


# rows of the sketch at 80 / 144 / 256 (the shapes' limits) and past them;
# columns: fewer than a warp's, one past a CTA's 16, one and several clusters,
# more than 32 columns on every SM (four lanes a column).
@pytest.mark.parametrize("m,n,nb,pp", [
    (60, 17, 8, 4), (90, 33, 16, 1), (200, 129, 70, 10), (200, 140, 71, 10), (400, 310, 134, 10),
    (400, 300, 135, 10), (700, 530, 246, 10), (300, 2433, 32, 10), (150, 5000, 60, 10),
    (260, 5100, 100, 10), (400, 5200, 200, 40), (40, 10000, 16, 8), (120, 9900, 90, 10)])
def test_plain_selection_shapes(hq, oracle_lib, m, n, nb, pp):
    _plain(hq, oracle_lib, m, n, nb, pp, m + n)


@pytest.mark.parametrize("nb,pp", [(64, 10), (128, 10), (200, 40)])
def test_mixed_selection_does_not_depend_on_the_layout(hq, nb, pp):
    """Zero columns appended to a matrix change the number of CTAs and which
    CTA a column lives in, never the pivots."""
    import torch
    m, n = 700, 600
    g = torch.Generator().manual_seed(nb)
    A = torch.randn(n, m, dtype=torch.float64, generator=g)
    hq.set_precision(hq.MIXED)
    got = []
    try:
        for extra in (0, 1, 700, 9000):
            At = torch.cat([A, torch.zeros(extra, m, dtype=torch.float64)]).cuda()
            jp = torch.arange(1, n + extra + 1, dtype=torch.int32, device="cuda")
            tau = torch.zeros(min(m, n + extra), dtype=torch.float64, device="cuda")
            hq.hqrrp_device(At, jp, tau, nb, pp, 1)
            got.append(jp[:nb].cpu().numpy())
    finally:
        hq.set_precision(hq.PLAIN)
    for other in got[1:]:
        np.testing.assert_array_equal(other, got[0])


def test_selection_reports_a_wait_that_gives_up(hq):
    """With a spin limit of 1 a poll gives up, the kernel ends with an error
    status and the next call is clean."""
    A = oracle.gaussian(400, 3000, 5)
    hq.set_precision(hq.PLAIN)
    want = hq.hqrrp(A, 64, 10, 1)
    hq.set_spin_limit(1)
    try:
        with pytest.raises(hq.HQRRPError, match="barrier"):
            hq.hqrrp(A, 64, 10, 1)
    finally:
        hq.set_spin_limit(0)
    got = hq.hqrrp(A, 64, 10, 1)
    for w, g in zip(want, got):
        np.testing.assert_array_equal(w, g)
