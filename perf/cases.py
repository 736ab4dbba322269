"""What this library is used for, as cases that can be timed and compared.

A case is a dict of plain values; its "kind" names the public call it makes:

  dgeqp4_host    hq.dgeqp4 on host (pageable numpy) arrays: the drop-in call
  dgeqp4_device  hq.dgeqp4_device on device arrays, free or partly fixed columns
  hqrrp          hq.hqrrp_device, the blocked factorization with its own nb
  batched        BatchedQRP.run, many uneven matrices in one launch (plan kept)
  truncated      hq.truncated_hqrrp, forward and backward through autograd
  apply_q        hq.apply_q: Q^T C of a factorization, as least squares needs it
  product        hq.ozaki_dgemm, the split-digit FP64 product on its own

Matrices are column-major on the device, so a (n, m) contiguous tensor.
Full factorizations get Gaussian columns of different lengths (columns in
different units, "decades" apart, in random order; 0 is plain i.i.d. N(0, 1));
the truncated and batched ones have singular values i^-2 with Haar factors.
"""
import math

import numpy as np
import torch

import hqrrp_gb300 as hq

PRECISION = {"plain": hq.PLAIN, "mixed": hq.MIXED}
F64 = torch.float64
BIG = 16384  # the largest factorization, the size the library is quoted on


def listed():
    return [
        # The drop-in call at its smallest: a dgeqp3 call site with a tiny
        # problem, where launches, allocations and copies are the time.
        {"name": "dgeqp4_host_96x64", "kind": "dgeqp4_host", "m": 96, "n": 64, "decades": 0.0,
         "precision": "plain"},
        # The dgeqp3 threshold branch (250 <= min(m, n) < 1000), odd sizes.
        {"name": "dgeqp4_641x481", "kind": "dgeqp4_device", "m": 641, "n": 481, "fixed": 0,
         "decades": 1.0, "precision": "plain"},
        # The HQRRP branch with some columns fixed by the caller.
        {"name": "dgeqp4_fixed_3001x2503", "kind": "dgeqp4_device", "m": 3001, "n": 2503,
         "fixed": 37, "decades": 2.0, "precision": "plain"},
        # The reference's own ordinary size and block: FP64, 2000^2, nb 64.
        {"name": "hqrrp_plain_2000", "kind": "hqrrp", "m": 2000, "n": 2000, "nb": 64, "pp": 10,
         "decades": 0.0, "precision": "plain"},
        # Mixed precision at an ordinary, ragged size.
        {"name": "hqrrp_mixed_3001x2999", "kind": "hqrrp", "m": 3001, "n": 2999, "nb": 128,
         "pp": 10, "decades": 1.0, "precision": "mixed"},
        # The largest: the size the headline is quoted on, mixed precision.
        {"name": "hqrrp_mixed_16384", "kind": "hqrrp", "m": BIG, "n": BIG, "nb": 128, "pp": 10,
         "decades": 2.0, "precision": "mixed"},
        # The drop-in call on a large tall host matrix, copies included.
        {"name": "dgeqp4_host_mixed_6144x3000", "kind": "dgeqp4_host", "m": 6144, "n": 3000,
         "decades": 1.0, "precision": "mixed"},
        # Many uneven small matrices, sizes log-uniform as in the benchmark.
        {"name": "batched_1024", "kind": "batched", "batch": 1024, "max_m": 1024, "max_n": 512},
        # The differentiable low-rank approximation: forward and backward, at
        # the benchmark's size in FP64 ...
        {"name": "truncated_plain_4096x2048", "kind": "truncated", "m": 4096, "n": 2048, "k": 256,
         "nb": 64, "precision": "plain"},
        # ... and wide, with a ragged rank, in mixed precision.
        {"name": "truncated_mixed_3000x5001", "kind": "truncated", "m": 3000, "n": 5001, "k": 200,
         "nb": 64, "precision": "mixed"},
        # Least squares after the factorization: Q^T times right-hand sides.
        {"name": "apply_qt_4001x1000", "kind": "apply_q", "m": 4001, "k": 1000, "nc": 72,
         "trans": "T", "precision": "plain"},
        # The product kernel of the mixed path called directly.
        {"name": "product_tn_4000", "kind": "product", "m": 4000, "n": 3001, "k": 4100,
         "ta": "T", "tb": "N", "slices": 7},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dgeqp4_host", "dgeqp4_small", "dgeqp4_large", "hqrrp", "hqrrp", "batched",
                       "truncated", "apply_q", "product"])
    precision = rng.choice(["plain", "mixed"])
    decades = round(rng.uniform(0.0, 2.0), 2)
    if kind == "dgeqp4_host":
        return {"kind": kind, "m": _log(rng, 16, 6144), "n": _log(rng, 16, 3000),
                "decades": decades, "precision": precision}
    if kind == "dgeqp4_small":  # min(m, n) < 1000, wide shapes among them
        m, n = _log(rng, 64, 999), _log(rng, 64, 3000)
        fixed = rng.choice([0, 0, 0, rng.randint(1, min(m, n) // 4)])
        return {"kind": "dgeqp4_device", "m": m, "n": n, "fixed": fixed, "decades": decades,
                "precision": precision}
    if kind == "dgeqp4_large":
        m, n = _log(rng, 1000, 4500), _log(rng, 1000, 4500)
        fixed = rng.choice([0, 0, rng.randint(1, 200)])
        return {"kind": "dgeqp4_device", "m": m, "n": n, "fixed": fixed, "decades": decades,
                "precision": precision}
    if kind == "hqrrp":
        top = 12288 if precision == "mixed" else 4096
        return {"kind": kind, "m": _log(rng, 500, top), "n": _log(rng, 500, top),
                "nb": rng.choice([64, 96, 128]), "pp": 10, "decades": decades,
                "precision": precision}
    if kind == "batched":
        return {"kind": kind, "batch": _log(rng, 64, 1024), "max_m": rng.choice([256, 512, 1024]),
                "max_n": rng.choice([128, 256, 512])}
    if kind == "truncated":
        return {"kind": kind, "m": _log(rng, 600, 6000), "n": _log(rng, 600, 6000),
                "k": _log(rng, 16, 300), "nb": rng.choice([64, 128]), "precision": precision}
    if kind == "apply_q":
        m = _log(rng, 300, 6000)
        return {"kind": kind, "m": m, "k": rng.randint(32, min(m, 1500)), "nc": _log(rng, 1, 1000),
                "trans": rng.choice("NT"), "precision": precision}
    return {"kind": kind, "m": _log(rng, 100, 5000), "n": _log(rng, 100, 5000),
            "k": _log(rng, 64, 6000), "ta": rng.choice("NT"), "tb": rng.choice("NT"),
            "slices": rng.choice([6, 7])}


# ---- Inputs ------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, dtype=F64, device="cuda", generator=g)


def _columns(m, n, decades, g):
    """A^T of an m x n Gaussian A whose columns' lengths span `decades`."""
    At = _randn(g, n, m)
    u = torch.rand(n, 1, dtype=F64, device="cuda", generator=g)
    return At.mul_(10.0 ** (-decades * u))


def _orthonormal(r, c, g):
    """r x c with Haar-distributed orthonormal columns: G chol(G^T G)^-T."""
    G = _randn(g, r, c)
    L = torch.linalg.cholesky(G.T @ G)
    return torch.linalg.solve_triangular(L, G.T, upper=False).T


def _spectrum(m, n, g):
    """A^T of A = U diag(i^-2) V^T."""
    k = min(m, n)
    s = torch.arange(1, k + 1, dtype=F64, device="cuda") ** -2.0
    return ((_orthonormal(n, k, g) * s) @ _orthonormal(m, k, g).T).contiguous()


def _shapes(case):
    """m log-uniform in [64, max_m], n log-uniform in [32, min(m, max_n)].
    The sizes belong to the plan, which a program keeps over its batches."""
    rng = np.random.default_rng(case["batch"] + case["max_m"] + case["max_n"])
    m = np.exp(rng.uniform(math.log(64), math.log(case["max_m"]), case["batch"])).astype(int)
    return [(int(a), int(math.exp(rng.uniform(math.log(32), math.log(min(a, case["max_n"]))))))
            for a in m]


def _batch(case, seed):
    g = _gen(seed)
    shapes = _shapes(case)
    offs = np.concatenate([[0], np.cumsum([m * n for m, n in shapes])]).astype(int)
    flat = torch.empty(int(offs[-1]), dtype=F64, device="cuda")
    for (m, n), o in zip(shapes, offs):
        flat[o:o + m * n].view(n, m).copy_(_spectrum(m, n, g))
    return shapes, offs, flat


def _fixed_marks(case, seed):
    """jpvt on entry of dgeqp4: `fixed` columns marked, at random places."""
    jp = np.zeros(case["n"], np.int32)
    if case.get("fixed"):
        jp[np.random.default_rng(seed).choice(case["n"], case["fixed"], replace=False)] = 1
    return jp


# ---- The cases ---------------------------------------------------------------

def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    s = {"case": case, "kind": kind, "precision": PRECISION[case.get("precision", "plain")]}
    if kind == "dgeqp4_host":
        s["A"] = np.asfortranarray(_columns(case["m"], case["n"], case["decades"], g).cpu().numpy().T)
    elif kind in ("dgeqp4_device", "hqrrp"):
        m, n = case["m"], case["n"]
        s["A"] = _columns(m, n, case["decades"], g)
        s["work"] = torch.empty_like(s["A"])
        jp = _fixed_marks(case, seed) if kind == "dgeqp4_device" else np.arange(1, n + 1, dtype=np.int32)
        s["jpvt_in"] = torch.from_numpy(jp).cuda()
        s["jpvt"] = torch.empty_like(s["jpvt_in"])
        s["tau"] = torch.zeros(min(m, n), dtype=F64, device="cuda")
    elif kind == "batched":
        shapes, offs, s["A"] = _batch(case, seed)
        s["work"] = torch.empty_like(s["A"])
        s["plan"] = hq.BatchedQRP(shapes)
        s["plan"].bind([s["work"][o:o + m * n].view(n, m) for (m, n), o in zip(shapes, offs)])
    elif kind == "truncated":
        s["A"] = _spectrum(case["m"], case["n"], g).t().requires_grad_()
        s["W"] = _randn(g, case["n"], case["m"]).t()
    elif kind == "apply_q":
        m, k = case["m"], case["k"]
        F, s["tau"] = torch.geqrf(_randn(g, m, k))
        s["F"] = F.t().contiguous()
        s["C"] = _randn(g, case["nc"], m)
        s["work"] = torch.empty_like(s["C"])
    else:
        s["X"], s["Y"] = _operands(case, g)
        s["out"] = torch.empty(case["n"], case["m"], dtype=F64, device="cuda")
    return s


def _operands(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    X = _randn(g, m, k) if case["ta"] == "T" else _randn(g, k, m)
    Y = _randn(g, k, n) if case["tb"] == "T" else _randn(g, n, k)
    return X, Y


def run(s):
    case, kind = s["case"], s["kind"]
    hq.set_precision(s["precision"])
    if kind == "dgeqp4_host":
        F, jpvt, tau, info, _ = hq.dgeqp4(s["A"])
        return F, jpvt, tau, info
    if kind == "dgeqp4_device":
        s["work"].copy_(s["A"])
        s["jpvt"].copy_(s["jpvt_in"])
        info = hq.dgeqp4_device(s["work"], s["jpvt"], s["tau"])
        return s["work"], s["jpvt"], s["tau"], info
    if kind == "hqrrp":
        s["work"].copy_(s["A"])
        s["jpvt"].copy_(s["jpvt_in"])
        hq.hqrrp_device(s["work"], s["jpvt"], s["tau"], case["nb"], case["pp"])
        return s["work"], s["jpvt"], s["tau"]
    if kind == "batched":
        s["work"].copy_(s["A"])
        s["plan"].run()
        return s["work"], s["plan"].jpvt_flat, s["plan"].tau_flat, s["plan"].info
    if kind == "truncated":
        A = s["A"]
        A.grad = None
        B = hq.truncated_hqrrp(A, case["k"], case["nb"])
        B.backward(s["W"])
        return B, A.grad
    if kind == "apply_q":
        s["work"].copy_(s["C"])
        return hq.apply_q(s["F"], s["tau"], s["work"], case["trans"], k=case["k"])
    hq.ozaki_dgemm(case["ta"], case["tb"], 1.0, s["X"], s["Y"], 0.0, s["out"], case["slices"])
    return s["out"]


def _qr_work(m, n):
    k, l = min(m, n), max(m, n)
    return {"bytes": 16.0 * m * n, "flops": 2.0 * l * k * k - 2.0 * k ** 3 / 3.0}


def work(case):
    kind = case["kind"]
    if kind in ("dgeqp4_host", "dgeqp4_device", "hqrrp"):
        return _qr_work(case["m"], case["n"])
    if kind == "batched":
        w = [_qr_work(m, n) for m, n in _shapes(case)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    if kind == "truncated":
        # Forward: the truncated factorization and one rank-k product.
        # Backward: Q (rebuilt), four m x n x k products and two k x k ones.
        m, n = case["m"], case["n"]
        k = min(case["k"], m, n)
        return {"bytes": 8.0 * 5 * m * n,
                "flops": 4.0 * m * n * k + 2.0 * m * n * k + 4.0 * m * k * k + 8.0 * m * n * k
                + 4.0 * m * k * k}
    if kind == "apply_q":
        m, k, nc = case["m"], case["k"], case["nc"]
        return {"bytes": 8.0 * (m * k + 2 * m * nc), "flops": (4.0 * m - 2.0 * k) * k * nc}
    m, n, k = case["m"], case["n"], case["k"]
    return {"bytes": 8.0 * (m * k + k * n + m * n), "flops": 2.0 * m * n * k}


# ---- What the outputs are in 64 bits, without this library --------------------

def _pivoted_qr(mats):
    """Column-pivoted Householder QR (LAPACK dgeqp3's output, all columns
    free) of a list of m x n matrices, zero-padded and worked on together:
    [(factored, jpvt, tau), ...]."""
    B, M = len(mats), max(a.shape[0] for a in mats)
    N = max(a.shape[1] for a in mats)
    X = torch.zeros(B, N, M, dtype=F64, device="cuda")  # column k of matrix i at X[i, k]
    for i, a in enumerate(mats):
        X[i, :a.shape[1], :a.shape[0]] = a.T
    ms = torch.tensor([a.shape[0] for a in mats], device="cuda")
    ns = torch.tensor([a.shape[1] for a in mats], device="cuda")
    steps = torch.minimum(ms, ns)
    at, cols = torch.arange(B, device="cuda"), torch.arange(N, device="cuda")
    perm = cols.repeat(B, 1)
    tau = torch.zeros(B, N, dtype=F64, device="cuda")
    for s in range(int(steps.max())):
        live = s < steps
        norms = X[:, s:, s:].square().sum(2)
        norms[cols[None, s:] >= ns[:, None]] = -1.0
        p = torch.where(live, norms.argmax(1) + s, s)
        for T in (X, perm):
            a, b = T[at, p].clone(), T[:, s].clone()
            T[:, s] = a
            T[at, p] = b
        x = X[:, s, s:]
        alpha, tail = x[:, 0].clone(), x[:, 1:].square().sum(1)
        beta = -torch.copysign(torch.sqrt(alpha * alpha + tail), alpha)
        none = (tail == 0) | ~live
        t = torch.where(none, 0.0, (beta - alpha) / torch.where(none, 1.0, beta))
        scale = torch.where(none, 0.0, 1.0 / torch.where(none, 1.0, alpha - beta))
        v = x * scale[:, None]
        v[:, 0] = 1.0
        w = torch.bmm(X[:, s + 1:, s:], v[:, :, None]) * t[:, None, None]
        X[:, s + 1:, s:].baddbmm_(w, v[:, None, :], alpha=-1.0)
        X[:, s, s] = torch.where(none, alpha, beta)
        X[:, s, s + 1:] = torch.where(none[:, None], X[:, s, s + 1:], v[:, 1:])
        tau[:, s] = t
    return [(X[i, :a.shape[1], :a.shape[0]], perm[i, :a.shape[1]].int() + 1,
             tau[i, :min(a.shape)]) for i, a in enumerate(mats)]


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind in ("dgeqp4_host", "dgeqp4_device"):
        # From 1000 on the pivots come from a random sketch: no one answer.
        if min(case["m"], case["n"]) >= 1000 or case.get("fixed"):
            return None
        At = _columns(case["m"], case["n"], case["decades"], g)
        F, jpvt, tau = _pivoted_qr([At.T])[0]
        return (F.T if kind == "dgeqp4_host" else F), jpvt, tau, None
    if kind == "batched":
        shapes, offs, flat = _batch(case, seed)
        done = _pivoted_qr([flat[o:o + m * n].view(n, m).T for (m, n), o in zip(shapes, offs)])
        return (torch.cat([F.reshape(-1) for F, _, _ in done]),
                torch.cat([jpvt for _, jpvt, _ in done]), torch.cat([t for _, _, t in done]), None)
    if kind == "apply_q":
        F, tau = torch.geqrf(_randn(g, case["m"], case["k"]))
        C = _randn(g, case["nc"], case["m"])
        return torch.ormqr(F, tau, C.T.contiguous(), left=True, transpose=case["trans"] == "T").T.contiguous()
    if kind == "product":
        X, Y = _operands(case, g)
        X = X if case["ta"] == "T" else X.T
        Y = Y.T if case["tb"] == "T" else Y
        return (X @ Y.T).T.contiguous()
    return None  # hqrrp, truncated: the pivots come from a random sketch
