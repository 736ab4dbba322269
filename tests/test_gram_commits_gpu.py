"""The mixed path's panels are the Gram panel's: what a call counts as committed
and as left to the cooperative panel kernel."""
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 2, 31, 32, 33, 63, 65, 96, 97, 127, 128])
def test_gaussian_panels_are_committed(hq, nb):
    m, n = 420, 290
    prev = hq.set_precision(hq.MIXED)
    try:
        hq.hqrrp(oracle.gaussian(m, n, nb), nb, 10, 1)
        counts = hq.gram_panel_counts()
    finally:
        hq.set_precision(prev)
    assert tuple(counts) == ((n + nb - 1) // nb, 0)
