"""The Gram panel's b x b kernels at the edges of their warps: block widths
around 32, 64, 96 and 128, with a ragged last block."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 2, 31, 32, 33, 63, 65, 96, 97, 127, 128])
def test_block_widths(hq, nb):
    m, n = 420, 290
    A = oracle.gaussian(m, n, nb)
    prev = hq.set_precision(hq.MIXED)
    try:
        before = hq.gram_panel_counts()
        Af, jpvt, tau = hq.hqrrp(A, nb, 10, 1)
        after = hq.gram_panel_counts()
    finally:
        hq.set_precision(prev)
    # A Gaussian panel is well conditioned: none falls back.
    assert after[1] == before[1] or after[1] == 0
    assert sorted(jpvt) == list(range(1, n + 1))
    res, orth, _ = oracle.quality(A, Af, jpvt, tau)
    assert res <= 1e-13 and orth <= 1e-12, (res, orth)
