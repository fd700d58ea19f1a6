"""Hessenberg reduction on the device (hsr_hessenberg_device) against LAPACK
dgehrd through scipy, the orthogonal factor it implies, extreme scalings, and
the dense-input pipeline: reduce, solve on H, back-transform."""
import numpy as np
import pytest

from hsrq3in_gb300 import generators as G

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _reduce(A):
    import torch
    import hsrq3in_gb300 as hsr
    n = A.shape[0]
    ld = n + 3                                                  # odd pitch on purpose
    dA = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
    dA[:, :n] = torch.from_numpy(np.ascontiguousarray(A.T))
    tau = hsr.hessenberg_device(dA)
    torch.cuda.synchronize()
    return dA, tau, dA[:, :n].cpu().numpy().T.copy(order="F"), tau.cpu().numpy()


def _form_q(dA, tau, n):
    import torch
    import hsrq3in_gb300 as hsr
    dQ = torch.eye(n, dtype=torch.float64, device="cuda")     # rows = columns of I
    hsr.hessenberg_apply_q_device(dA, tau, dQ)
    torch.cuda.synchronize()
    return dQ.cpu().numpy().T


@pytest.mark.parametrize("n,seed", [(1, 1), (2, 2), (3, 3), (4, 4), (17, 5), (100, 6), (300, 7), (700, 8)])
def test_matches_lapack_dgehrd(gpu_lib, n, seed):
    from scipy.linalg import lapack
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((n, n))
    _, _, out, tau = _reduce(A)
    hq, tau_ref, info = lapack.dgehrd(np.asfortranarray(A))
    assert info == 0
    scale = np.linalg.norm(A)
    np.testing.assert_allclose(np.triu(out, -1), np.triu(hq, -1), rtol=0, atol=1e3 * n * EPS * scale)
    np.testing.assert_allclose(tau[:n - 1], tau_ref[:n - 1], rtol=0, atol=1e3 * n * EPS)
    np.testing.assert_allclose(np.tril(out, -2), np.tril(hq, -2), rtol=0, atol=1e3 * n * EPS)


@pytest.mark.parametrize("n", [50, 400])
def test_q_orthogonal_similarity(gpu_lib, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    dA, tau, out, _ = _reduce(A)
    H = np.triu(out, -1)
    Q = _form_q(dA, tau, n)
    assert np.linalg.norm(Q.T @ Q - np.eye(n)) <= 50 * n * EPS
    assert np.linalg.norm(A @ Q - Q @ H) / np.linalg.norm(A) <= 50 * n * EPS


@pytest.mark.parametrize("scale", [1e300, 1e-300])
def test_extreme_scale(gpu_lib, scale):
    from scipy.linalg import lapack
    rng = np.random.default_rng(9)
    n = 120
    A = rng.standard_normal((n, n))
    _, _, out, _ = _reduce(A * scale)
    assert np.all(np.isfinite(out))
    hq, _, _ = lapack.dgehrd(np.asfortranarray(A))
    np.testing.assert_allclose(np.triu(out, -1) / scale, np.triu(hq, -1), rtol=0,
                               atol=1e3 * n * EPS * np.linalg.norm(A))


def test_dense_pipeline(gpu_lib):
    """Dense A with a known real spectrum: reduce on the device, solve on H,
    back-transform with Q; every eigenpair of A within the residual bound."""
    import torch
    import hsrq3in_gb300 as hsr
    n = 600
    H0, lam = G.real_spectrum(n, 21)
    rng = np.random.default_rng(22)
    Z, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = Z @ H0 @ Z.T
    dA, tau, out, _ = _reduce(A)
    H = np.triu(out, -1)
    wr = G.perturbed_shifts(lam, 23)
    sol = hsr.inverse_iteration(np.asfortranarray(H), wr, 64, 64)
    dX = torch.from_numpy(np.ascontiguousarray(sol["vr"].T)).cuda()
    hsr.hessenberg_apply_q_device(dA, tau, dX)
    torch.cuda.synchronize()
    X = dX.cpu().numpy().T
    R = A @ X - X * sol["wr"][None, :]
    res = np.linalg.norm(R, axis=0) / (np.linalg.norm(A) * np.linalg.norm(X, axis=0))
    assert np.all(res <= 100 * n * EPS), res.max()


@pytest.mark.parametrize("n,scale,leading", [(5, 1e-300, 0), (60, 1e-300, 0), (60, 1e-305, 1), (300, 1e-300, 2),
                                             (60, 1.0, 1)])
def test_zero_subdiagonal_at_the_safe_minimum(gpu_lib, n, scale, leading):
    """Columns whose reflector starts from an exact 0 above entries that need
    the safe-minimum rescaling: `leading` columns that are zero below the
    diagonal, then one with a zero on the subdiagonal.  A Q = Q H and Q^T Q = I
    with Q formed in extended precision, to within n eps as 2n Householder
    transformations leave it."""
    L = np.longdouble
    A = np.random.default_rng(n + leading).standard_normal((n, n))
    for k in range(leading):
        A[k + 1:, k] = 0.0
    A[leading + 1, leading] = 0.0
    _, _, F, tau = _reduce(A * scale)
    Q = np.eye(n, dtype=L)
    for k in range(n - 3, -1, -1):
        v = F[k + 1:, k].astype(L)
        v[0] = 1.0
        Q[k + 1:] -= np.outer(v, tau[k] * (v[:, None] * Q[k + 1:]).sum(0))
    G = np.array([(Q * Q[:, c:c + 1]).sum(0) for c in range(n)]) - np.eye(n)
    assert float(np.sqrt((G * G).sum())) <= n * EPS * np.sqrt(n)
    H = np.triu(F, -1).astype(L) / scale
    R = np.array([(A * Q[:, c]).sum(1) - (Q[:, :c + 2] * H[:c + 2, c]).sum(1) for c in range(n)])
    assert float(np.sqrt((R * R).sum())) <= n * EPS * np.linalg.norm(A)


@pytest.mark.parametrize("n,scale,graded", [(3, 1.0, False), (64, 1.0, False), (67, 1e-300, False), (130, 1.0, True),
                                            (300, 1e150, False), (300, 1.0, True), (2100, 1.0, False)])
def test_three_launches_a_column(gpu_lib, monkeypatch, n, scale, graded):
    """The forms for orders whose panel does not fit one launch and for devices
    that refuse a cooperative one, forced: A Q = Q H and Q^T Q = I, with a zero
    on the subdiagonal of A's first column; graded: the updates in FP64 too."""
    import torch
    import hsrq3in_gb300 as hsr
    monkeypatch.setenv("HSR_HESS_PANEL", "steps")
    A = np.random.default_rng(n).standard_normal((n, n))
    A[1, 0] = 0.0
    if graded:
        A *= 10.0 ** (-9 * np.arange(n) / n)
    dA, tau, out, _ = _reduce(A * scale)
    one = hsr.hessenberg_device(torch.zeros_like(dA))           # and of a zero matrix
    assert not torch.any(one)
    Q = torch.from_numpy(_form_q(dA, tau, n)).cuda()
    H, At = torch.from_numpy(np.triu(out, -1) / scale).cuda(), torch.from_numpy(A).cuda()
    assert float((Q.T @ Q - torch.eye(n, dtype=torch.float64, device="cuda")).norm()) <= 50 * n * EPS
    assert float((At @ Q - Q @ H).norm()) / np.linalg.norm(A) <= 50 * n * EPS
