"""Digit products on the tensor cores (hsr_digits.cuh) where they can go wrong:
sizes at the edges of their tiles (128 rows, 64 columns, 16 and 192 inner),
graded and non-finite inputs.  Each is compared with the same formula in
extended precision; tolerances follow from the FP64 operations that remain
around the exact digit sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _cols(torch, A, pad):
    """Columns of A as rows of a device tensor with a padded leading dimension."""
    out = torch.full((A.shape[1], A.shape[0] + pad), 5.0, dtype=torch.float64, device="cuda")
    out[:, :A.shape[0]] = torch.from_numpy(np.ascontiguousarray(A.T))
    return out


@pytest.mark.parametrize("n,ncols,pad,graded", [
    (127, 3, 0, False), (128, 64, 1, False), (129, 65, 0, False), (191, 1, 3, False), (193, 63, 0, False),
    (255, 130, 1, False), (385, 70, 0, True), (640, 33, 2, True)])
def test_residuals_against_extended(gpu_lib, n, ncols, pad, graded):
    """Every operation after the exact products rounds once in FP64: the sum
    of n squares and the two norms, at most n eps / 2 each, and a few more."""
    import torch
    import hsrq3in_gb300 as hsr
    rng = np.random.default_rng(n)
    H = rng.standard_normal((n, n))
    X = rng.standard_normal((n, ncols))
    if graded:                                   # columns of H over 60 decades, x the other way
        d = 10.0 ** rng.uniform(-30, 30, n)
        H, X = H * d, X / d[:, None]
    wr = rng.uniform(-2, 2, ncols)
    got = hsr.residuals_device(_cols(torch, H, pad), torch.from_numpy(wr).cuda(), _cols(torch, X, pad)).cpu().numpy()
    L = np.longdouble
    Hh, Xl = np.triu(H, -1).astype(L), X.astype(L)
    R = np.array([(Hh * Xl[:, c]).sum(1) for c in range(ncols)]).T - Xl * wr.astype(L)
    ref = np.sqrt((R * R).sum(0)) / (np.sqrt((Hh * Hh).sum()) * np.sqrt((Xl * Xl).sum(0)))
    np.testing.assert_allclose(got, ref.astype(np.float64), rtol=(2 * n + 32) * EPS)


def test_residuals_non_finite(gpu_lib):
    """A column of x with an Inf or a NaN gives NaN, a zero one Inf, the others
    their value; garbage below the subdiagonal of H does not enter."""
    import torch
    import hsrq3in_gb300 as hsr
    n = 300
    rng = np.random.default_rng(1)
    H, X, wr = rng.standard_normal((n, n)), rng.standard_normal((n, 5)), rng.uniform(-1, 1, 5)
    X[7, 1], X[299, 2], X[:, 3] = np.inf, np.nan, 0.0
    H[np.tril_indices(n, -2)] = np.nan
    got = hsr.residuals_device(_cols(torch, H, 0), torch.from_numpy(wr).cuda(), _cols(torch, X, 1)).cpu().numpy()
    Hh = np.triu(H, -1)
    for c in (0, 4):
        ref = np.linalg.norm(Hh @ X[:, c] - wr[c] * X[:, c]) / (np.linalg.norm(Hh) * np.linalg.norm(X[:, c]))
        np.testing.assert_allclose(got[c], ref, rtol=1e-12)
    assert np.isnan(got[1]) and np.isnan(got[2]) and np.isposinf(got[3])
    H[5, 200] = np.inf
    assert np.isnan(hsr.residuals_device(_cols(torch, H, 0), torch.from_numpy(wr).cuda(),
                                         _cols(torch, X, 0)).cpu().numpy()[[0, 1, 2, 4]]).all()


def _reflectors(rng, n):
    """(A, tau): random Householder vectors as hsr_hessenberg_device leaves them."""
    A = rng.standard_normal((n, n))
    tau = np.zeros(n)
    for k in range(n - 2):
        x = A[k + 1:, k]
        beta = -np.copysign(np.linalg.norm(x), x[0])
        tau[k] = (beta - x[0]) / beta
        A[k + 2:, k] /= x[0] - beta
    return A, tau


@pytest.mark.parametrize("n,ncols,pad", [(40, 1, 0), (127, 63, 1), (128, 64, 0), (129, 65, 3), (130, 3, 0),
                                         (131, 130, 0), (258, 16, 1), (259, 5, 0), (515, 70, 0)])
def test_back_transform_against_extended(gpu_lib, n, ncols, pad):
    """Reflector by reflector in extended precision; n Householder reflectors
    in FP64 are within n eps of it, column by column."""
    import torch
    import hsrq3in_gb300 as hsr
    rng = np.random.default_rng(n)
    A, tau = _reflectors(rng, n)
    X = rng.standard_normal((n, ncols)) * 10.0 ** rng.uniform(-200, 200, ncols)
    dX = _cols(torch, X, pad)
    hsr.hessenberg_apply_q_device(_cols(torch, A, pad), torch.from_numpy(tau).cuda(), dX)
    R = X.astype(np.longdouble)
    for k in range(n - 3, -1, -1):
        v = A[k + 1:, k].astype(np.longdouble)
        v[0] = 1.0
        R[k + 1:] -= np.outer(v, tau[k] * (v[:, None] * R[k + 1:]).sum(0))
    got = dX.cpu().numpy()
    err = np.sqrt((((got[:, :n].T - R) / np.abs(R).max(0)) ** 2).sum(0)) / np.sqrt(((R / np.abs(R).max(0)) ** 2).sum(0))
    assert err.max() <= n * EPS, err.max()
    assert np.all(got[:, n:] == 5.0)


def test_back_transform_non_finite(gpu_lib):
    """An Inf or NaN in a column of X spoils that column's rows from 1 on, as
    the reflectors do one by one, and no other column."""
    import torch
    import hsrq3in_gb300 as hsr
    n = 200
    rng = np.random.default_rng(3)
    A, tau = _reflectors(rng, n)
    X = rng.standard_normal((n, 4))
    ref = _cols(torch, X, 0)
    hsr.hessenberg_apply_q_device(_cols(torch, A, 0), torch.from_numpy(tau).cuda(), ref)
    X[60, 1], X[150, 2] = np.nan, np.inf
    dX = _cols(torch, X, 0)
    hsr.hessenberg_apply_q_device(_cols(torch, A, 0), torch.from_numpy(tau).cuda(), dX)
    got, ref = dX.cpu().numpy(), ref.cpu().numpy()
    assert np.array_equal(got[[0, 3]], ref[[0, 3]])
    assert not np.isfinite(got[1:3, 1:]).any() and np.array_equal(got[1:3, 0], X[0, 1:3])


@pytest.mark.parametrize("n,pad,scale", [(32, 0, 1.0), (66, 1, 1e150), (67, 0, 1.0), (130, 0, 1e-150), (193, 3, 1.0),
                                         (258, 0, 1.0), (322, 1, 1e8)])
def test_reduction_backward_error(gpu_lib, n, pad, scale):
    """A = Q H Q^T to within n eps |A|, the backward error of 2n Householder
    transformations, with Q formed in extended precision from the reflectors."""
    import torch
    import hsrq3in_gb300 as hsr
    A = np.random.default_rng(n).standard_normal((n, n))
    dA = _cols(torch, A * scale, pad)
    tau = hsr.hessenberg_device(dA).cpu().numpy()
    got = dA.cpu().numpy()
    assert np.all(got[:, n:] == 5.0)
    F = got[:, :n].T
    Q = np.eye(n, dtype=np.longdouble)
    for k in range(n - 3, -1, -1):
        v = F[k + 1:, k].astype(np.longdouble)
        v[0] = 1.0
        Q[k + 1:] -= np.outer(v, tau[k] * (v[:, None] * Q[k + 1:]).sum(0))
    H = np.triu(F, -1).astype(np.longdouble) / scale
    R = np.array([(A * Q[:, c]).sum(1) - (Q[:, :c + 2] * H[:c + 2, c]).sum(1) for c in range(n)])   # A Q - Q H
    err = float(np.sqrt((R * R).sum()))
    assert err <= n * EPS * np.linalg.norm(A), (err, np.linalg.norm(A))


def test_reduction_nan_in_first_row(gpu_lib):
    """Row 0 takes no part in any reflector: a NaN there stays in that row and
    the rest is what it is without it."""
    import torch
    import hsrq3in_gb300 as hsr
    n = 150
    A = np.random.default_rng(5).standard_normal((n, n))
    clean = _cols(torch, A, 0)
    tau = hsr.hessenberg_device(clean)
    A[0, 100] = np.nan
    got = _cols(torch, A, 0)
    tau2 = hsr.hessenberg_device(got)
    assert torch.equal(tau, tau2) and torch.equal(got[:, 1:], clean[:, 1:])
    assert torch.isnan(got[1:, 0]).all()


@pytest.mark.parametrize("n,pad,scale,graded", [(2048, 0, 1.0, False), (2051, 1, 1e-290, False), (2112, 0, 1e280, True),
                                                (2400, 0, 1.0, True)])
def test_reduction_fixed_point_panel(gpu_lib, n, pad, scale, graded):
    """Orders whose panels multiply by the matrix in fixed point: A Q = Q H to
    within n eps |A| (as above, Q from the back-transform of the identity),
    also with rows and columns of very different size."""
    import torch
    import hsrq3in_gb300 as hsr
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    if graded:
        A *= 10.0 ** rng.uniform(-6, 0, n)[:, None] * 10.0 ** rng.uniform(-6, 0, n)
    dA = _cols(torch, A * scale, pad)
    tau = hsr.hessenberg_device(dA)
    Q = torch.eye(n, dtype=torch.float64, device="cuda")
    hsr.hessenberg_apply_q_device(dA, tau, Q)                    # rows = columns of Q
    Q = Q.T
    H = torch.triu(dA[:, :n].T, -1) / scale
    R = torch.from_numpy(A).cuda() @ Q - Q @ H
    assert float(R.norm()) <= n * EPS * np.linalg.norm(A)


def test_reduction_fixed_point_non_finite(gpu_lib):
    """A NaN in row 0 stays there; an Inf elsewhere reaches what it reaches
    with products in floating point."""
    import torch
    import hsrq3in_gb300 as hsr
    n = 2050
    A = np.random.default_rng(2).standard_normal((n, n))
    ref = _cols(torch, A, 0)
    tref = hsr.hessenberg_device(ref)
    A[0, 1000] = np.nan
    dA = _cols(torch, A, 0)
    tau = hsr.hessenberg_device(dA)
    assert torch.equal(dA[:, 1:], ref[:, 1:]) and torch.equal(tau, tref)
    A[0, 1000], A[700, 1200] = 0.0, np.inf
    dA = _cols(torch, A, 0)
    hsr.hessenberg_device(dA)
    assert not torch.isfinite(dA[2:, 1:2]).any()


def test_reductions_on_two_streams(gpu_lib):
    """One thread, two streams, no wait between the calls: each reduction and
    back-transform (with digits, and small enough to go without) gives what it
    gives alone."""
    import torch
    import hsrq3in_gb300 as hsr
    rng = np.random.default_rng(8)
    for n in (20, 300):
        A = [rng.standard_normal((n, n)) for _ in range(6)]
        X = rng.standard_normal((n, 7))
        ref = []
        for a in A:
            d, x = _cols(torch, a, 0), _cols(torch, X, 0)
            t = hsr.hessenberg_device(d)
            hsr.hessenberg_apply_q_device(d, t, x)
            ref.append((d, t, x))
        st = [torch.cuda.Stream(), torch.cuda.Stream()]
        got = [(_cols(torch, a, 0), _cols(torch, X, 0)) for a in A]
        torch.cuda.synchronize()
        tau = []
        for i, (d, x) in enumerate(got):
            with torch.cuda.stream(st[i & 1]):
                tau.append(hsr.hessenberg_device(d, stream=st[i & 1]))
                hsr.hessenberg_apply_q_device(d, tau[-1], x, stream=st[i & 1])
        torch.cuda.synchronize()
        for (d, x), t, (rd, rt, rx) in zip(got, tau, ref):
            assert torch.equal(d, rd) and torch.equal(t, rt) and torch.equal(x, rx)


def test_back_transform_sum_below_power_of_two(gpu_lib):
    """An update whose exact sum lies 2^-53 below 4: five reflectors meet in
    row 150 with (2^-27, 1, 1, 1, 1) (-2^-26, 1, 1, 1, 1)^T, the rest of the
    block is the identity and the first block random.  Tolerance as above."""
    import torch
    import hsrq3in_gb300 as hsr
    n, r = 160, 150
    A, tau = _reflectors(np.random.default_rng(4), n)
    A[:, 128:] = np.triu(A, -1)[:, 128:]
    tau[128:] = 0.0
    tau[128:133] = 1.0
    A[r, 128:133] = [2.0 ** -27, 1, 1, 1, 1]
    X = np.zeros((n, 2))
    X[129:134, 0] = [2.0 ** -26, 4, 3, 2, 1]
    X[129:134, 1] = [-2.0 ** -26, -4, -3, -2, -1]
    dX = _cols(torch, X, 0)
    hsr.hessenberg_apply_q_device(_cols(torch, A, 0), torch.from_numpy(tau).cuda(), dX)
    R = X.astype(np.longdouble)
    for k in range(n - 3, -1, -1):
        v = A[k + 1:, k].astype(np.longdouble)
        v[0] = 1.0
        R[k + 1:] -= np.outer(v, tau[k] * (v[:, None] * R[k + 1:]).sum(0))
        if k == 128:
            assert np.array_equal(R[r], np.longdouble([-1, 1]) * (4 - np.longdouble(2) ** -53))
    err = np.sqrt(((dX.cpu().numpy().T - R) ** 2).sum(0)) / np.sqrt((R * R).sum(0))
    assert err.max() <= n * EPS, err.max()


@pytest.mark.parametrize("n", [40, 200, 389])
def test_back_transform_first_row(gpu_lib, n):
    """Row 0 takes part in no reflector: whatever is there, the other rows are
    what they are without it, bit for bit, and it stays."""
    import torch
    import hsrq3in_gb300 as hsr
    rng = np.random.default_rng(n)
    A, tau = _reflectors(rng, n)
    dA, dtau = _cols(torch, A, 0), torch.from_numpy(tau).cuda()
    X = np.repeat(rng.standard_normal((n, 1)), 5, axis=1)
    X[0] = [0.5, 1e20, -1e300, np.inf, np.nan]
    dX = _cols(torch, X, 1)
    hsr.hessenberg_apply_q_device(dA, dtau, dX)
    got = dX.cpu().numpy()
    assert np.isfinite(got[0]).all() and np.array_equal(got[:, 0], X[0], equal_nan=True)
    for c in range(1, 5):
        assert np.array_equal(got[c, 1:n], got[0, 1:n]), c


def _form_q(torch, F, tau):
    """Q of the reflectors in F (columns as usual) and tau, one by one in FP64."""
    n = F.shape[0]
    Q = torch.eye(n, dtype=torch.float64, device="cuda")
    for k in range(n - 3, -1, -1):
        v = F[k + 1:, k].clone()
        v[0] = 1.0
        Q[k + 1:] -= tau[k] * torch.outer(v, v @ Q[k + 1:])
    return Q


def _reduce_one_by_one(torch, A):
    """dgehd2 in FP64: the reflectors one by one."""
    F, n = A.clone(), A.shape[0]
    tau = torch.zeros(n, dtype=torch.float64, device="cuda")
    for k in range(n - 2):
        x = F[k + 1:, k].clone()
        if not torch.any(x[1:]):
            continue                             # tau = 0
        beta = -torch.copysign(torch.linalg.norm(x), x[0])
        tau[k] = (beta - x[0]) / beta
        v = x / (x[0] - beta)
        v[0] = 1.0
        F[:, k + 1:] -= tau[k] * torch.outer(F[:, k + 1:] @ v, v)
        F[k + 1:, k + 1:] -= tau[k] * torch.outer(v, v @ F[k + 1:, k + 1:])
        F[k + 1, k] = beta
        F[k + 2:, k] = v[1:]
    return F, tau


@pytest.mark.parametrize("n,pad,decades", [(33, 0, 10), (130, 1, 16), (160, 0, 30), (300, 0, 12), (2100, 0, 16),
                                           (160, 0, 2.4), (300, 1, 3.6), (2100, 0, 2.4)])   # near where FP64 takes over
def test_reduction_keeps_graded_rows(gpu_lib, n, pad, decades):
    """A = D G D with D falling over many decades: the Householder reduction in
    FP64 keeps the small rows and columns, (Q^T A Q - H)_ij of the size of d_i
    d_j eps.  Within ten times of the reflectors one by one in FP64, whose sums
    run in another order; a window below the largest entry would lose
    everything (1e9 times and more)."""
    import torch
    import hsrq3in_gb300 as hsr
    d = 10.0 ** (-decades * np.arange(n) / (n - 1))
    A = np.random.default_rng(n).standard_normal((n, n)) * d[:, None] * d
    dA = _cols(torch, A, pad)
    tau = hsr.hessenberg_device(dA)
    assert torch.all(dA[:, n:] == 5.0)
    At, D = torch.from_numpy(A).cuda(), torch.from_numpy(d).cuda()
    err = []
    for F, t in ((dA[:, :n].T.contiguous(), tau), _reduce_one_by_one(torch, At)):
        Q = _form_q(torch, F, t)
        err.append(float(((Q.T @ At @ Q - torch.triu(F, -1)) / D[:, None] / D).abs().max()))
    assert err[0] <= 10 * err[1], err


@pytest.mark.parametrize("n,pad", [(32, 0), (65, 1), (130, 0), (321, 3), (2049, 0)])
@pytest.mark.parametrize("form", ["zero", "eye", "band", "permutation", "sparse", "hessenberg", "blocks", "even"])
def test_reduction_of_any_form(gpu_lib, n, pad, form):
    """Matrices that the digit products take and that they leave to FP64: A Q =
    Q H and Q^T Q = I to within n eps as in test_reduction_backward_error."""
    import torch
    import hsrq3in_gb300 as hsr
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    if form == "zero":
        A[:] = 0.0
    elif form == "eye":
        A = np.eye(n) + 1e-9 * A
    elif form == "band":
        A = np.tril(np.triu(A, -3), 2)
    elif form == "permutation":
        A = np.eye(n)[rng.permutation(n)]
    elif form == "sparse":
        A *= rng.random((n, n)) < 0.1
    elif form == "hessenberg":
        A = np.triu(A, -1)
    elif form == "blocks":
        A[: n // 2, n // 2:] *= 1e9
        A[n // 2:, : n // 2] *= 1e-9
    else:
        A = rng.uniform(0.0, 1.0, (n, n))
    dA = _cols(torch, A, pad)
    tau = hsr.hessenberg_device(dA)
    F = dA[:, :n].T.contiguous()
    At, Q = torch.from_numpy(A).cuda(), _form_q(torch, F, tau)
    assert float((Q.T @ Q - torch.eye(n, dtype=torch.float64, device="cuda")).norm()) <= n * EPS * np.sqrt(n)
    assert float((At @ Q - Q @ torch.triu(F, -1)).norm()) <= n * EPS * np.linalg.norm(A)


@pytest.mark.parametrize("n,ncols,pad,decades", [(45, 3, 0, 8), (130, 65, 1, 10), (200, 5, 0, 25), (300, 30, 0, 12),
                                                 (200, 30, 0, 1.8), (300, 5, 0, 2.4)])   # near where FP64 takes over
def test_back_transform_keeps_graded_rows(gpu_lib, n, ncols, pad, decades):
    """Reflectors of a graded matrix on columns graded alike: FP64 keeps the
    small rows.  Row by row, relative to the row's largest entry, within ten
    times of the reflectors one by one in FP64, whose sums run in another
    order; both against extended precision."""
    import torch
    import hsrq3in_gb300 as hsr
    rng = np.random.default_rng(n)
    d = 10.0 ** (-decades * np.arange(n) / (n - 1))
    F, tau = _reduce_one_by_one(torch, torch.from_numpy(rng.standard_normal((n, n)) * d[:, None] * d).cuda())
    A, tau = F.cpu().numpy(), tau.cpu().numpy()
    X = rng.standard_normal((n, ncols)) * d[:, None]
    dX = _cols(torch, X, pad)
    hsr.hessenberg_apply_q_device(_cols(torch, A, pad), torch.from_numpy(tau).cuda(), dX)
    got = dX.cpu().numpy()
    assert np.all(got[:, n:] == 5.0)
    R, S = X.astype(np.longdouble), X.copy()
    for k in range(n - 3, -1, -1):
        v = A[k + 1:, k].copy()
        v[0] = 1.0
        S[k + 1:] -= np.outer(v, tau[k] * (v[:, None] * S[k + 1:]).sum(0))
        v = v.astype(np.longdouble)
        R[k + 1:] -= np.outer(v, tau[k] * (v[:, None] * R[k + 1:]).sum(0))
    scale = np.abs(R).max(1)[:, None]
    err = [float((np.abs(Z - R) / scale).max()) for Z in (got[:, :n].T, S)]
    assert err[0] <= 10 * err[1], err


@pytest.mark.parametrize("n,ncols", [(40, 1), (65, 64), (130, 65), (321, 7)])
@pytest.mark.parametrize("form", ["identity", "hessenberg", "band", "sparse", "first", "late"])
def test_back_transform_of_any_form(gpu_lib, n, ncols, form):
    """Reflectors that the digit products take and that they leave to FP64, and
    columns of one large entry: within n eps of extended precision, column by
    column, as in test_back_transform_against_extended."""
    import torch
    import hsrq3in_gb300 as hsr
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n))
    X = rng.standard_normal((n, ncols))
    if form == "identity":
        M[np.tril_indices(n, -2)] = 0.0
    elif form == "hessenberg":
        M[np.tril_indices(n, -2)] *= 1e-14
    elif form == "band":
        M = np.tril(M, 3)
    elif form == "sparse":
        M *= rng.random((n, n)) < 0.2
    elif form == "first":
        X[2:] *= 1e-25
    else:
        X[: n // 2] = 0.0
    F, tau = _reduce_one_by_one(torch, torch.from_numpy(M).cuda())
    A, tau = F.cpu().numpy(), tau.cpu().numpy()
    dX = _cols(torch, X, 0)
    hsr.hessenberg_apply_q_device(_cols(torch, A, 0), torch.from_numpy(tau).cuda(), dX)
    R = X.astype(np.longdouble)
    for k in range(n - 3, -1, -1):
        v = A[k + 1:, k].astype(np.longdouble)
        v[0] = 1.0
        R[k + 1:] -= np.outer(v, tau[k] * (v[:, None] * R[k + 1:]).sum(0))
    err = np.sqrt(((dX.cpu().numpy().T - R) ** 2).sum(0)) / np.sqrt((R * R).sum(0))
    assert err.max() <= n * EPS, err.max()
