"""The pivoted panel kernel's source, run on the CPU with its warps in one order
and in the opposite one: every shared word is read after the barrier that
follows its write, so the two give the same bits -- and LAPACK's factorization.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hqrrp_gb300", "csrc")


@pytest.fixture(scope="module")
def panel(tmp_path_factory):
    from hqrrp_gb300 import buildlib
    cuda = buildlib.cuda_home()
    out = tmp_path_factory.mktemp("panel")
    with open(os.path.join(CSRC, "qrp_panel.cu")) as f:
        text = f.read()
    begin, end = text.index("namespace {"), text.index("\nint panel_grid(")
    decl = "extern __shared__ __align__(16) double smem[];"
    kernel = text[begin:end]
    assert kernel.count(decl) == 1
    kernel = '#include "hq_fixedpoint.h"\n' + kernel.replace(decl, "double* smem = emu_smem;") + "\n}\n"
    (out / "panel_kernel.inc").write_text(kernel)
    lib = str(out / "libpanel.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-shared", "-fPIC", "-I", str(out), "-I", CSRC,
                    "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "panel_harness.cpp"), "-o", lib], check=True)
    so = C.CDLL(lib)
    so.hq_test_panel.argtypes = [C.c_int] * 5 + [C.c_void_p] * 4

    def run(A, order, pivoting=1, smem_mode=1):
        m, n = A.shape
        F = np.asfortranarray(A.copy())
        tau, perm, nbar = np.zeros(min(m, n)), np.zeros(n, np.int32), C.c_int()
        rc = so.hq_test_panel(m, n, pivoting, smem_mode, order, F.ctypes.data, tau.ctypes.data,
                              perm.ctypes.data, C.addressof(nbar))
        assert rc == 0
        return F, tau, perm, nbar.value
    run.so = so
    return run


@pytest.mark.parametrize("smem_mode", [1, 0])
@pytest.mark.parametrize("m,n", [(40, 24), (30, 40), (70, 128), (20, 130), (9, 33), (200, 40),
                                 (300, 140), (193, 60)])
def test_any_order_of_the_warps(panel, m, n, smem_mode):
    import scipy.linalg as sl
    rng = np.random.default_rng(m + n)
    # Columns of very different lengths: the pivots are far from their places.
    A = np.asfortranarray(rng.standard_normal((m, n)) * 10.0 ** rng.uniform(-8, 8, n))
    F, tau, perm, _ = panel(A, 0, smem_mode=smem_mode)
    F1, tau1, perm1, _ = panel(A, 1, smem_mode=smem_mode)
    np.testing.assert_array_equal(perm, perm1)
    np.testing.assert_array_equal(tau, tau1)
    np.testing.assert_array_equal(F, F1)
    (_, to), Ro, po = sl.qr(A, mode="raw", pivoting=True)
    np.testing.assert_array_equal(perm, po)
    np.testing.assert_allclose(tau, to, atol=1e-12)
    k = min(m, n)
    R, Rr = np.triu(F[:k]), np.triu(Ro[:k])
    assert np.max(np.linalg.norm(R - Rr, axis=0) / np.linalg.norm(Rr, axis=0)) <= 1e-12


@pytest.mark.parametrize("smem_mode", [1, 0])
@pytest.mark.parametrize("pivoting", [1, 0])
def test_any_order_with_recomputed_norms(panel, pivoting, smem_mode):
    rng = np.random.default_rng(5)
    m, n = 60, 50
    A = np.asfortranarray(rng.standard_normal((m, 4)) @ rng.standard_normal((4, n))
                          + rng.standard_normal((m, n)) * 10.0 ** -rng.uniform(5.0, 6.0, n))
    F, tau, perm, barriers = panel(A, 0, pivoting, smem_mode)
    assert barriers == 1 if not pivoting else barriers > 1
    for a, b in zip((F, tau, perm), panel(A, 1, pivoting, smem_mode)):
        np.testing.assert_array_equal(a, b)
    Q = np.eye(m)
    for k in reversed(range(n)):
        v = np.concatenate([np.zeros(k), [1.0], F[k + 1:, k]])
        Q -= tau[k] * np.outer(v, v @ Q)
    assert np.linalg.norm(Q @ np.triu(F) - A[:, perm]) <= 1e-13 * np.linalg.norm(A)


def test_a_norm_is_recomputed_only_when_it_has_cancelled(panel):
    cancelled = panel.so.hq_test_norm_cancelled
    cancelled.argtypes = [C.c_double] * 2
    inf, nan = np.inf, np.nan
    for nd, thr in ((0.5, 1.0), (1.0, 1.0), (0.0, 0.0), (-0.0, 1e-300), (-3.0, 1.0), (-inf, 1.0)):
        assert cancelled(nd, thr)
    for nd, thr in ((2.0, 1.0), (1e-300, 0.0), (inf, 1.0), (inf, inf), (nan, 1.0), (nan, nan),
                    (-nan, 1.0), (-nan, nan), (-nan, -nan), (nan, inf)):
        assert not cancelled(nd, thr)


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e200])
@pytest.mark.parametrize("smem_mode", [1, 0])
def test_a_norm_that_is_not_finite_is_not_recomputed(panel, bad, smem_mode):
    """Nor are the other columns': one grid barrier, for the initial norms."""
    rng = np.random.default_rng(2)
    m, n = 40, 24
    A = np.asfortranarray(rng.standard_normal((m, n)))
    A[7, 5] = bad
    F, tau, perm, barriers = panel(A, 0, smem_mode=smem_mode)
    assert barriers == 1 and sorted(perm) == list(range(n))
    assert not np.all(np.isfinite(F))
