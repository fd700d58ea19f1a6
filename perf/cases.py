"""The work that programs give this framework, as timed cases.

A case names one call (or one plan's execution) with its sizes:

* ``drop_in``  tiled_inverse_iteration on host arrays, as a C or numpy caller
  of the reference makes it
* ``solve``    the same solve on device-resident tensors, all or some shifts,
  with the library's start vectors or the caller's right-hand sides
* ``cplx``     complex-conjugate shifts on device-resident tensors
* ``batch``    a plan over many small problems of uneven order and shift count
* ``served``   the request loop on host buffers, all requests waiting
* ``hess``     reduction of a dense matrix to Hessenberg form
* ``back``     back-transform of vectors with the reduction's orthogonal factor
* ``resid``    residuals of approximate eigenpairs

``listed`` spans the range of each; ``draw`` gives more of the same ranges.
"""
import math

import numpy as np
import torch

import hsrq3in_gb300 as hsr

DEV = "cuda"
F64 = torch.float64
ULP = 2.0 ** -53


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A program with a small matrix: one call on host arrays, where the
        # launches, copies and synchronisations are most of the time.
        dict(name="drop_in_n48", kind="drop_in", n=48, nrhs=48, tlsz=16),
        # The usual drop-in call: a few thousand rows, half of the spectrum.
        dict(name="drop_in_n2000", kind="drop_in", n=2000, nrhs=1000, tlsz=160),
        # The benchmark's small plain configuration, device-resident.
        dict(name="solve_n1000", kind="solve", n=1000, nrhs=1000, tlsz=160, scaling="pow2", user_rhs=False),
        # Part of the spectrum of a larger matrix, an odd order and shift
        # count, caller's right-hand sides, the reference's scaling factors.
        dict(name="solve_n3001_part", kind="solve", n=3001, nrhs=301, tlsz=200, scaling="double", user_rhs=True),
        # The benchmark's large plain configuration: all 10,000 eigenvectors.
        dict(name="solve_n10000", kind="solve", n=10000, nrhs=10000, tlsz=160, scaling="pow2", user_rhs=False),
        # Complex eigenvalues of a real matrix, a part of the pairs.
        dict(name="cplx_n2000", kind="cplx", n=2000, pairs=500, tlsz=160),
        # The benchmark's batch: orders log-uniform in [32, 1024], a quarter
        # to all of the eigenvalues each.
        dict(name="batch_192", kind="batch", count=192, nlo=32, nhi=1024, mix=1),
        # The request loop with a burst of mixed requests.
        dict(name="served_40", kind="served", count=40, nlo=64, nhi=1500, mix=2),
        # Dense inputs: reduction of a small and of a large matrix.
        dict(name="hess_n700", kind="hess", n=700),
        dict(name="hess_n6000", kind="hess", n=6000),
        # Eigenvectors of the dense matrix from those of H.
        dict(name="back_n5000", kind="back", n=5000, ncols=2500),
        # Checking approximate eigenpairs before they are used or refined.
        dict(name="resid_n5000", kind="resid", n=5000, ncols=5000),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drop_in", "solve", "cplx", "batch", "served", "hess", "back", "resid"])
    part = lambda n, lo=0.05: max(1, int(round(n * math.exp(rng.uniform(math.log(lo), 0.0)))))  # noqa: E731
    tlsz = rng.choice([64, 96, 128, 160, 200])
    if kind == "drop_in":
        n = _logint(rng, 32, 3000)
        return dict(kind=kind, n=n, nrhs=part(n), tlsz=tlsz if n > 300 else 16)
    if kind == "solve":
        n = _logint(rng, 200, 7000)
        return dict(kind=kind, n=n, nrhs=part(n), tlsz=tlsz, scaling=rng.choice(["pow2", "double"]),
                    user_rhs=rng.random() < 0.3)
    if kind == "cplx":
        n = _logint(rng, 200, 3500)
        return dict(kind=kind, n=n, pairs=max(1, part(n) // 2), tlsz=tlsz)
    if kind == "batch":
        return dict(kind=kind, count=_logint(rng, 48, 256), nlo=32, nhi=rng.choice([128, 300, 1024]),
                    mix=rng.randrange(1 << 20))
    if kind == "served":
        return dict(kind=kind, count=_logint(rng, 12, 60), nlo=64, nhi=rng.choice([300, 1500]),
                    mix=rng.randrange(1 << 20))
    if kind == "hess":
        return dict(kind=kind, n=_logint(rng, 200, 6500))
    if kind == "back":
        n = _logint(rng, 400, 6500)
        return dict(kind=kind, n=n, ncols=part(n, 0.02))
    n = _logint(rng, 300, 6500)
    return dict(kind=kind, n=n, ncols=part(n, 0.02))


def _mix(case):
    """Orders and shift counts of a batch or a request mix."""
    r = np.random.default_rng(case["mix"])
    ns = np.exp(r.uniform(np.log(case["nlo"]), np.log(case["nhi"]), case["count"])).round().astype(int)
    return [(int(n), max(1, int(round(n * f)))) for n, f in zip(ns, r.uniform(0.25, 1.0, case["count"]))]


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _similar(g, B):
    """triu(R B R^-1, -1) for a random unit upper-triangular R: Hessenberg,
    dense above the diagonal, non-normal, with the eigenvalues of the
    Hessenberg matrix B of bandwidth two.  Returns (H, R)."""
    n = B.shape[0]
    R = torch.triu(_randn(g, n, n).mul_(3.5 / math.sqrt(n)), 1)
    R.diagonal().fill_(1.0)
    d0, dl, du = B.diagonal().clone(), B.diagonal(-1).clone(), B.diagonal(1).clone()
    H = R * d0
    H[:, :-1] += R[:, 1:] * dl
    H[:, 1:] += R[:, :-1] * du
    torch.linalg.solve_triangular(R, H, upper=True, left=False, unitriangular=True, out=H)
    return H.triu_(-1), R


def _grid(g, m):
    """m distinct values in [-1, 1] on a jittered grid, in random order."""
    lam = -1.0 + (2.0 / m) * (torch.arange(m, device=DEV, dtype=F64) + 0.5 + 0.5 * (_rand(g, m) - 0.5))
    return lam[torch.randperm(m, generator=g, device=DEV)]


def _offset(g, H, m):
    """Distances of shifts from their eigenvalues: what a backward-stable
    eigenvalue solver leaves, of the size of the rounding of H, either sign."""
    norm = float(H.abs().sum(1).max())
    return torch.sign(_rand(g, m) - 0.5) * (0.125 + 0.125 * _rand(g, m)) * (ULP * norm)


def _real(g, n):
    """(H, eigenvalues, R, the lower bidiagonal B with H = R B R^-1)."""
    B = torch.diag(_grid(g, n))
    if n > 1:
        B.diagonal(-1).copy_(0.04 + 0.08 * _rand(g, n - 1))
    H, R = _similar(g, B)
    return H, B.diagonal().clone(), R, B


def _real_problem(g, n, m):
    H, lam, _, _ = _real(g, n)
    at = torch.sort(torch.randperm(n, generator=g, device=DEV)[:m]).values
    return H, lam[at] + _offset(g, H, m)


def _complex_problem(g, n, m):
    p = n // 2
    a = _grid(g, p)
    b = 0.1 + 0.9 * _rand(g, p)
    d, up, lo = torch.zeros(n, device=DEV, dtype=F64), torch.zeros(n - 1, device=DEV, dtype=F64), 0.04 + 0.08 * _rand(g, n - 1)
    d[0:2 * p:2], d[1:2 * p:2] = a, a
    if n % 2:
        d[n - 1] = 2.0
    up[0:2 * p:2], lo[0:2 * p:2] = b, -b
    H, _ = _similar(g, torch.diag(d) + torch.diag(up, 1) + torch.diag(lo, -1))
    at = torch.sort(torch.randperm(p, generator=g, device=DEV)[:m]).values
    return H, a[at] + _offset(g, H, m), b[at] + _offset(g, H, m)


def _columns(H):
    """H as the device entry points take it: rows of the tensor are columns,
    an even leading dimension."""
    n = H.shape[0]
    out = torch.zeros(n, n + (n & 1), device=DEV, dtype=F64)
    out[:, :n] = H.T
    return out


def _even(n):
    return n + (n & 1)


def _inputs(case, seed):
    """What a solve takes, as plain matrices: [(H, wr)], [(H, wr, rhs)] or
    [(H, wr, wi)]."""
    g, kind = _gen(seed), case["kind"]
    if kind == "cplx":
        return [_complex_problem(g, case["n"], case["pairs"])]
    if kind in ("batch", "served"):
        return [_real_problem(g, n, m) for n, m in _mix(case)]
    H, wr = _real_problem(g, case["n"], case["nrhs"])
    return [(H, wr, _rand(g, case["nrhs"], case["n"]))] if case.get("user_rhs") else [(H, wr)]


def _dense_reflectors(g, n):
    """(A, tau) with Householder vectors below the subdiagonal as a reduction
    of a random matrix leaves them."""
    A = _randn(g, n, n)                                     # A[i, j]: row i, column j
    x = torch.tril(A, -2)
    alpha = A.diagonal(-1)
    norm = torch.sqrt((x * x).sum(0)[: n - 1] + alpha * alpha)
    beta = -torch.copysign(norm, alpha)
    x[:, : n - 1] /= alpha - beta
    tau = torch.zeros(n, device=DEV, dtype=F64)
    tau[: n - 1] = (beta - alpha) / beta
    tau[n - 2:] = 0.0
    return torch.triu(A, -1) + x, tau


def _near_eigenpairs(g, n, m):
    """(H, wr, X): eigenpairs of H to about five digits, X's rows the vectors."""
    H, lam, R, B = _real(g, n)
    at = torch.randperm(n, generator=g, device=DEV)[:m]
    V = torch.zeros(m, n, device=DEV, dtype=F64)
    V[torch.arange(m, device=DEV), at] = 1.0
    ratio = torch.zeros(m, n, device=DEV, dtype=F64)
    ratio[:, 1:] = B.diagonal(-1) / (lam[at][:, None] - lam[None, 1:])
    below = torch.arange(n, device=DEV)[None, :] > at[:, None]
    V = torch.where(below, torch.cumprod(torch.where(below, ratio, torch.ones_like(ratio)), 1), V)
    X = V @ R.T
    X /= torch.linalg.norm(X, dim=1, keepdim=True)
    X += 1e-5 / math.sqrt(n) * _randn(g, m, n)
    return H, lam[at], X


def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"], "tlsz": case.get("tlsz")}
    if kind in ("drop_in", "solve", "cplx", "batch", "served"):
        probs = _inputs(case, seed)
    if kind == "drop_in":
        H, wr = probs[0]
        s.update(H=np.asfortranarray(H.cpu().numpy()), wr=wr.cpu().numpy())
    elif kind == "solve":
        H, wr = probs[0][:2]
        n, m = H.shape[0], wr.numel()
        s.update(H=_columns(H), wr0=wr, wr=wr.clone(), X=torch.zeros(m, _even(n), device=DEV, dtype=F64), n=n,
                 scaling=case["scaling"], rhs=probs[0][2] if case["user_rhs"] else None,
                 status=torch.zeros(m, device=DEV, dtype=torch.int32),
                 scale=torch.zeros(m, device=DEV, dtype=F64))
    elif kind == "cplx":
        H, wr, wi = probs[0]
        s.update(H=_columns(H), wr=wr, wi=wi, X=torch.zeros(2 * wr.numel(), _even(H.shape[0]), device=DEV, dtype=F64),
                 status=torch.zeros(wr.numel(), device=DEV, dtype=torch.int32))
    elif kind == "batch":
        s["wr0"] = torch.cat([wr for _, wr in probs])
        s["wr"] = s["wr0"].clone()
        s["X"] = torch.zeros(sum(wr.numel() * _even(H.shape[0]) for H, wr in probs), device=DEV, dtype=F64)
        at, wat, list_ = 0, 0, []
        for H, wr in probs:
            m, ld = wr.numel(), _even(H.shape[0])
            list_.append((_columns(H), s["wr"][wat:wat + m], s["X"][at:at + m * ld].view(m, ld)))
            at, wat = at + m * ld, wat + m
        s["plan"] = hsr.BatchPlan(list_)
    elif kind == "served":
        size = sum(wr.numel() * H.shape[0] for H, wr in probs)
        out = torch.zeros(size, dtype=F64).pin_memory()
        s.update(out=out, server=hsr.Server(hbm_budget_bytes=8e9), reqs=[], wr0=[], keep=[])
        at = 0
        for H, wr in probs:
            n, m = H.shape[0], wr.numel()
            Hh = torch.empty(n, n, dtype=F64).pin_memory()
            Hh.copy_(H.T)
            w = wr.cpu().pin_memory()
            s["keep"].append((Hh, w))
            s["wr0"].append(w.numpy().copy())
            s["reqs"].append(dict(H=Hh.numpy().T, wr=w.numpy(), vr=out[at:at + n * m].view(m, n).numpy().T,
                                  arrival_s=0.0))
            at += n * m
    elif kind == "hess":
        n = case["n"]
        s.update(A0=_randn(_gen(seed), n, n), A=torch.zeros(n, n, device=DEV, dtype=F64))
    elif kind == "back":
        g = _gen(seed)
        A, tau = _dense_reflectors(g, case["n"])
        s.update(A=A.T.contiguous(), tau=tau, X0=_randn(g, case["ncols"], case["n"]))
        s["X"] = torch.zeros_like(s["X0"])
    else:
        H, wr, X = _near_eigenpairs(_gen(seed), case["n"], case["ncols"])
        s.update(H=_columns(H), wr=wr, X=X)
    return s


# --------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "drop_in":
        vr, wr = hsr.tiled_inverse_iteration(s["H"], s["wr"], s["tlsz"], 64)
        return {"vr": vr, "wr": wr}
    if kind == "solve":
        s["wr"].copy_(s["wr0"])                              # a restart may reorder the shifts
        if s["rhs"] is not None:
            s["X"][:, :s["n"]].copy_(s["rhs"])
        rc = hsr.inverse_iteration_device(s["H"], s["wr"], s["X"], s["tlsz"], scaling=s["scaling"],
                                          user_rhs=s["rhs"] is not None, d_status=s["status"], d_scale=s["scale"])
        return {"vr": s["X"], "wr": s["wr"], "status": s["status"], "scale": s["scale"], "rc": rc}
    if kind == "cplx":
        rc = hsr.inverse_iteration_cplx_device(s["H"], s["wr"], s["wi"], s["X"], s["tlsz"], d_status=s["status"])
        return {"vr": s["X"], "status": s["status"], "rc": rc}
    if kind == "batch":
        s["wr"].copy_(s["wr0"])
        rc = s["plan"].execute()
        return {"vr": s["X"], "wr": s["wr"], "rc": rc}
    if kind == "served":
        for r, w in zip(s["reqs"], s["wr0"]):
            r["wr"][:] = w
        _, status, _ = s["server"].replay(s["reqs"])
        return {"vr": s["out"], "status": np.array(status)}
    if kind == "hess":
        s["A"].copy_(s["A0"])                                # the reduction is in place; A is kept for checks
        tau = hsr.hessenberg_device(s["A"])
        return {"A": s["A"], "tau": tau}
    if kind == "back":
        s["X"].copy_(s["X0"])
        hsr.hessenberg_apply_q_device(s["A"], s["tau"], s["X"])
        return {"X": s["X"]}
    return {"res": hsr.residuals_device(s["H"], s["wr"], s["X"])}


def work(case):
    """Inputs read once and outputs written once; the operations of the
    algorithm: n^2 per shift for the crossover columns and n^2 for the
    updates (twice that in complex arithmetic), 10/3 n^3 for the reduction,
    2 n^2 per vector for the back-transform, n^2 per vector for a residual."""
    kind = case["kind"]

    def solve(n, m, rhs=False):
        return 8.0 * (n * n / 2 + n * m * (2 if rhs else 1) + 2 * m), 2.0 * n * n * m

    if kind in ("drop_in", "solve"):
        b, f = solve(case["n"], case["nrhs"], case.get("user_rhs", False))
    elif kind == "cplx":
        n, p = case["n"], case["pairs"]
        b, f = 8.0 * (n * n / 2 + 2 * n * p + 2 * p), 4.0 * n * n * p
    elif kind in ("batch", "served"):
        each = [solve(n, m) for n, m in _mix(case)]
        b, f = sum(x for x, _ in each), sum(x for _, x in each)
    elif kind == "hess":
        n = case["n"]
        b, f = 16.0 * n * n, 10.0 / 3.0 * n ** 3
    elif kind == "back":
        n, m = case["n"], case["ncols"]
        b, f = 8.0 * (n * n / 2 + 2 * n * m), 2.0 * n * n * m
    else:
        n, m = case["n"], case["ncols"]
        b, f = 8.0 * (n * n / 2 + n * m + 2 * m), 1.0 * n * n * m
    return {"bytes": b, "flops": f}


# ------------------------------------------------- the same in plain torch
def _vectors(H, mu, rhs=None):
    """Unit vectors (rows) along (H - mu_k)^-1 b_k, and the growth of each:
    the RQ factorisation of the shifted matrices by plane rotations of
    columns, all shifts at once, with the back-substitution beside it."""
    n, m = H.shape[0], mu.numel()
    Hc = H.T.contiguous().to(mu.dtype)                       # rows are columns of H
    v = Hc[n - 1].repeat(m, 1)
    v[:, n - 1] -= mu
    b = torch.ones(m, n, device=DEV, dtype=mu.dtype) if rhs is None else rhs.to(mu.dtype).clone()
    b0 = torch.linalg.norm(b, dim=1)
    z = torch.zeros(n, m, device=DEV, dtype=mu.dtype)
    cs, sn = torch.zeros(n, m, device=DEV, dtype=mu.dtype), torch.zeros(n, m, device=DEV, dtype=mu.dtype)
    for j in range(n - 1, 0, -1):
        col = Hc[j - 1, : j + 1].repeat(m, 1)
        col[:, j - 1] -= mu
        g, t = col[:, j], v[:, j]
        r = torch.sqrt(t.abs() ** 2 + g.abs() ** 2)
        cs[j], sn[j] = t / r, g / r
        c, s = cs[j][:, None], sn[j][:, None]
        z[j] = b[:, j] / r
        b[:, :j] -= z[j][:, None] * (s.conj() * col[:, :j] + c.conj() * v[:, :j])
        v = c * col[:, :j] - s * v[:, :j]
    z[0] = b[:, 0] / v[:, 0]
    for j in range(1, n):
        lo, hi = z[j - 1].clone(), z[j].clone()
        z[j - 1] = cs[j] * lo + sn[j].conj() * hi
        z[j] = cs[j].conj() * hi - sn[j] * lo
    norm = torch.linalg.norm(z, dim=0)
    return (z / norm).T, norm / b0


def _settled(H, growth):
    """Whether every vector grows enough in one solve (start vectors of the
    size of H's rounding, growth to 0.1 / sqrt(n)), with a margin."""
    n = H.shape[0]
    eps3 = ULP * float(H.abs().sum(1).max())
    return bool((growth * eps3 * math.sqrt(n) > 0.3 / math.sqrt(n)).all())


def _padded(X, ld):
    out = torch.zeros(X.shape[0], ld, device=DEV, dtype=F64)
    out[:, : X.shape[1]] = X
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("drop_in", "solve", "batch", "served"):
        rows, shifts = [], []
        for p in _inputs(case, seed):
            H, wr = p[:2]
            X, growth = _vectors(H, wr, p[2] if len(p) > 2 else None)
            if len(p) == 2 and not _settled(H, growth):
                return None                                  # a restart changes that vector's sign and place
            rows.append(X)
            shifts.append(wr)
        if kind == "drop_in":
            return {"vr": rows[0].T.cpu().numpy(), "wr": shifts[0]}
        if kind == "served":
            return {"vr": torch.cat([x.reshape(-1) for x in rows]), "status": None}
        if kind == "batch":
            return {"vr": torch.cat([_padded(x, _even(x.shape[1])).reshape(-1) for x in rows]),
                    "wr": torch.cat(shifts), "rc": None}
        return {"vr": _padded(rows[0], _even(case["n"])), "wr": shifts[0], "status": None, "scale": None, "rc": None}
    if kind == "cplx":
        H, wr, wi = _inputs(case, seed)[0]
        X, growth = _vectors(H, torch.complex(wr, wi))
        if not _settled(H, growth):
            return None
        out = torch.zeros(2 * wr.numel(), case["n"], device=DEV, dtype=F64)
        out[0::2], out[1::2] = X.real, X.imag
        return {"vr": _padded(out, _even(case["n"])), "status": None, "rc": None}
    if kind == "hess":
        n = case["n"]
        A = _randn(_gen(seed), n, n)                         # row k is column k
        tau = torch.zeros(n, device=DEV, dtype=F64)
        for k in range(n - 2):
            x = A[k, k + 1:]
            beta = -torch.copysign(torch.linalg.norm(x), x[0])
            tau[k] = (beta - x[0]) / beta
            v = x / (x[0] - beta)
            v[0] = 1.0
            rest = A[k + 1:]
            rest -= tau[k] * torch.outer(v, v @ rest)
            low = A[k + 1:, k + 1:]
            low -= tau[k] * torch.outer(low @ v, v)
            A[k, k + 1] = beta
            A[k, k + 2:] = v[1:]
        return {"A": A, "tau": tau}
    if kind == "back":
        g = _gen(seed)
        A, tau = _dense_reflectors(g, case["n"])
        X = _randn(g, case["ncols"], case["n"])
        for k in range(case["n"] - 3, -1, -1):
            v = A[k + 1:, k].clone()
            v[0] = 1.0
            low = X[:, k + 1:]
            low -= torch.outer(low @ v, tau[k] * v)
        return {"X": X}
    H, wr, X = _near_eigenpairs(_gen(seed), case["n"], case["ncols"])
    r = X @ H.T - wr[:, None] * X
    return {"res": torch.linalg.norm(r, dim=1) / (torch.linalg.norm(H) * torch.linalg.norm(X, dim=1))}
