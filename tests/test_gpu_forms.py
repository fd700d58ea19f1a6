"""The forms of the diagonal solve, of the top rows' GEMM and of the
finalisation that a solve takes by its number of shifts and its tile height,
each against the oracle: bit for bit, so there is no tolerance."""
import numpy as np
import pytest

from hsrq3in_gb300 import generators as G
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tlsz,pairs", [
    (40, 16, 1), (40, 16, 3), (72, 20, 17),       # 4 pairs per CTA, its remainders
    (64, 16, 700), (130, 48, 1203),               # 8
    (64, 24, 1300), (47, 16, 2430),               # 16
    (64, 16, 2500),                               # a warp's 32 lanes
    (210, 200, 700), (210, 200, 1300),            # a tile high for the narrow forms
    (400, 392, 600), (400, 392, 2500),            # one that needs the global scratch in the wide form
])
def test_complex_forms(gpu_lib, n, tlsz, pairs):
    import hsrq3in_gb300 as hsr
    H, lam, _ = G.complex_spectrum(n, n + pairs)
    mu = np.resize(lam, pairs)
    dev = hsr.inverse_iteration_cplx(H, mu, tlsz, 16)
    orc = O.oracle_inverse_iteration_cplx(H, mu.real, mu.imag, tlsz, 16, intscale=1, variant="fma")
    assert np.array_equal(dev["vr"], orc["vr"])
    assert np.array_equal(dev["perturbed"], orc["perturbed"])
    assert np.array_equal(dev["scale"], orc["colscale"])
    assert np.array_equal(dev["status"], orc["status"])


@pytest.mark.parametrize("n,shifts", [
    (1, 1), (2, 33), (15, 1), (16, 31), (17, 32), (31, 33), (32, 64), (33, 65),   # blocks of 16 rows, 32 columns
    (48, 607), (48, 609), (50, 1215), (50, 1217), (49, 2431), (49, 2433),         # 4, 8, 16 shifts per CTA, or 32
])
@pytest.mark.parametrize("tlsz", [8, 16])
def test_real_forms(gpu_lib, n, tlsz, shifts):
    import hsrq3in_gb300 as hsr
    H, lam = G.real_spectrum(n, n + shifts)
    wr = np.resize(G.perturbed_shifts(lam, 3), shifts)
    dev = hsr.inverse_iteration(H, wr, tlsz, 16)
    orc = O.oracle_inverse_iteration(H, wr, tlsz, 16, intscale=1, variant="fma")
    assert np.array_equal(dev["vr"], orc["vr"])
    assert np.array_equal(dev["perturbed"], orc["perturbed"])
    assert np.array_equal(dev["scale"], orc["colscale"])
    assert np.array_equal(dev["status"], orc["status"])


@pytest.mark.parametrize("scaling,intscale", [("pow2", 1), ("double", 0)])
def test_upscaled_tiles(gpu_lib, scaling, intscale):
    """Tiles whose scaling factors differ: the back-transform multiplies a
    tile's rows before their rotations."""
    import hsrq3in_gb300 as hsr
    H, sh = G.block_scaled(96, 16, 3)
    sh = np.asarray(sh)[:5]
    for cplx in (False, True):
        if cplx:
            mu = sh + 1e-3j
            dev = hsr.inverse_iteration_cplx(H, mu, 16, 4, scaling=scaling, max_restarts=1)
            orc = O.oracle_inverse_iteration_cplx(H, mu.real, mu.imag, 16, 16, intscale=intscale, max_restarts=1,
                                                  variant="fma")
        else:
            dev = hsr.inverse_iteration(H, sh, 16, 4, scaling=scaling)
            orc = O.oracle_inverse_iteration(H, sh, 16, 16, intscale=intscale, variant="fma")
        assert np.array_equal(dev["vr"], orc["vr"], equal_nan=True)
        assert np.array_equal(dev["scale"], orc["colscale"], equal_nan=True)
        assert np.array_equal(dev["status"], orc["status"])


@pytest.mark.parametrize("count,tlsz", [(1, 64), (9, 16), (19, 32), (20, 64), (30, 16), (60, 32), (60, 100)])
def test_batch_forms(gpu_lib, count, tlsz):
    """Batches whose ticks take 4, 8 and 16 shifts per CTA, down to the last
    problem's: each problem as the oracle solves it."""
    import torch
    import hsrq3in_gb300 as hsr
    probs, ref = [], []
    for i in range(count):
        n = 1 + (37 * i + 100) % 150
        H, lam = G.real_spectrum(n, i + 1)
        wr = np.resize(G.perturbed_shifts(lam, i), (11 * i) % 70 + 1)
        ld = n + (n & 1)
        Hd = torch.zeros((n, ld), dtype=torch.float64)
        Hd[:, :n] = torch.from_numpy(H.T.copy())
        probs.append((Hd.cuda()[:, :n], torch.from_numpy(wr.copy()).cuda(),
                      torch.zeros((wr.size, ld), dtype=torch.float64, device="cuda")))
        ref.append(O.oracle_inverse_iteration(H, wr, tlsz, 16, intscale=1, variant="fma"))
    plan = hsr.BatchPlan(probs, tlsz=tlsz)
    plan.execute()
    for (H, _, X), o in zip(probs, ref):
        assert np.array_equal(X.cpu().numpy()[:, :H.shape[0]].T, o["vr"])
    plan.close()


@pytest.mark.parametrize("n,tlsz,nrhs", [(203, 40, 77), (260, 160, 609), (300, 64, 1217)])
def test_forced_shifts_per_cta(gpu_lib, monkeypatch, n, tlsz, nrhs):
    """A forced number of shifts per diagonal CTA is the one that runs: the
    kernels' instantiation shows in a trace, the result is the oracle's."""
    import torch
    import hsrq3in_gb300 as hsr
    from torch.profiler import ProfilerActivity, profile
    H, lam = G.real_spectrum(n, n)
    wr = np.resize(G.perturbed_shifts(lam, 3), nrhs)
    orc = O.oracle_inverse_iteration(H, wr, tlsz, 16, intscale=1, variant="fma")
    for sc in (4, 8, 16, 32):
        monkeypatch.setenv("HSR_DIAG_SHIFTS_PER_CTA", str(sc))
        for _ in range(2):                       # a process's first trace can come back empty
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                dev = hsr.inverse_iteration(H, wr, tlsz, 16)
                torch.cuda.synchronize()
            names = [e.key for e in prof.key_averages()]
            diag = [k for k in names if "k_diag" in k]
            if diag:
                break
        if not any("k_" in k for k in names):
            pytest.skip("no kernel trace on this machine")
        assert diag and all(("k_diag_n" in k and "<%d, " % sc in k) if sc < 32 else "k_diag_n" not in k for k in diag), (sc, diag)
        assert np.array_equal(dev["vr"], orc["vr"])
