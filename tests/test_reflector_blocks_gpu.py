"""The triangular factor of a reflector block, Q formed from the unit columns,
and the adjoint's triangular solve, at the edges of their warps and blocks."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _t(A):
    import torch
    return torch.from_numpy(np.ascontiguousarray(A.T)).cuda()


def _reflectors(m, k, seed):
    """Random reflectors, every seventh the identity (tau = 0)."""
    rng = np.random.default_rng(seed)
    F = rng.standard_normal((m, k)) / np.sqrt(m)
    V = np.tril(F, -1) + np.eye(m, k)
    tau = 2.0 / np.sum(V * V, axis=0)
    tau[6::7] = 0.0
    return F, V, tau


@pytest.mark.parametrize("m,k,nb", [
    (1, 1, 1), (40, 5, 1), (70, 31, 31), (70, 64, 32), (200, 100, 33), (400, 300, 128),
    (400, 260, 129), (300, 255, 255), (400, 300, 256), (300, 270, 200), (129, 129, 64),
])
def test_form_and_apply_q(hq, m, k, nb):
    import torch
    F, V, tau = _reflectors(m, k, m + k + nb)
    tt = torch.from_numpy(tau).cuda()
    rng = np.random.default_rng(1)
    C = rng.standard_normal((m, 17))
    Q, QC, QtC = np.eye(m, k), C.copy(), C.copy()
    for i in range(k):
        QtC -= tau[i] * np.outer(V[:, i], V[:, i] @ QtC)
        j = k - 1 - i
        Q -= tau[j] * np.outer(V[:, j], V[:, j] @ Q)
        QC -= tau[j] * np.outer(V[:, j], V[:, j] @ QC)
    # k reflectors, each with a product of length m, on columns of norm 1 (C's: sqrt(m)).
    tol = 10 * (m + k) * 2.0 ** -53
    got = hq.form_q(_t(F), tt, k, nb).cpu().numpy().T
    assert np.abs(got - Q).max() <= tol
    for trans, ref in (("N", QC), ("T", QtC)):
        Ct = _t(C)
        out = hq.apply_q(_t(F), tt, Ct, trans, k, nb)
        got = (Ct if out is None else out).cpu().numpy().T
        assert np.abs(got - ref).max() <= tol * np.sqrt(m)


@pytest.mark.parametrize("m,n,k", [(100, 80, 1), (100, 80, 31), (97, 120, 32), (100, 80, 33),
                                   (161, 130, 65), (33, 40, 33)])
def test_adjoint_at_solve_block_edges(hq, m, n, k):
    import torch
    rng = np.random.default_rng(m + n + k)
    A = oracle.with_spectrum(m, n, (1.0 + np.arange(min(m, n))) ** -2.0, m + k)
    W = rng.standard_normal((m, n))
    At = _t(A)
    Ft, jp, tau = hq.truncated_factor(At, k, 32)
    G = hq.adjoint(At, Ft, jp, tau, _t(W), k, 32).cpu().numpy().T
    perm = jp.cpu().numpy() - 1
    X = torch.tensor(A, dtype=torch.float64, requires_grad=True)
    Q, _ = torch.linalg.qr(X[:, perm[:k]])
    (torch.tensor(W) * (Q @ (Q.T @ X))).sum().backward()
    ref = X.grad.numpy()
    assert np.linalg.norm(G - ref) <= 1e-10 * np.linalg.norm(ref)
