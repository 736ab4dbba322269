"""The FP64 GEMM at the edges of its 16 x 16 parts and 32 x 32 tiles, with and
without slices of K, through the blocked reflector application (a Gram matrix
of which only the upper triangle is formed, U^T C, op(T) W and C - U W)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# m, k, nb, nc: one row / column short of, at and past a part and a tile; K
# (the rows) below one step, and long enough to be cut; more columns than rows.
SHAPES = [(17, 16, 16, 15), (33, 31, 31, 32), (48, 33, 33, 33), (65, 64, 64, 1), (97, 17, 1, 80),
          (2049, 65, 64, 47), (4097, 96, 96, 31), (1500, 74, 74, 1201), (31, 5, 7, 3000)]


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("m,k,nb,nc", SHAPES)
def test_reflector_application_at_tile_edges(hq, m, k, nb, nc, trans):
    import scipy.linalg as sl
    import torch
    rng = np.random.default_rng(m + 31 * k + nc)
    A, C = rng.standard_normal((m, k)), rng.standard_normal((m, nc))
    (F, tau), _ = sl.qr(A, mode="raw")
    # Q C one reflector at a time, in extended precision where the host has it.
    want = C.astype(np.longdouble)
    order = range(k) if trans == "T" else range(k - 1, -1, -1)
    for j in order:
        v = np.zeros(m, np.longdouble)
        v[j] = 1.0
        v[j + 1:] = F[j + 1:, j]
        want -= tau[j] * np.outer(v, v @ want)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    Ct = dev(C.T)
    hq.set_precision(hq.PLAIN)
    hq.apply_q(dev(F.T), dev(tau), Ct, trans, k, nb)
    # Backward error of a product of k reflectors: a few k eps of each column.
    bound = 10.0 * k * np.finfo(float).eps * np.linalg.norm(C, axis=0)
    err = np.linalg.norm((Ct.cpu().numpy().T - want).astype(float), axis=0)
    assert np.all(err <= np.maximum(bound, 1e-14)), float(np.max(err / bound))
