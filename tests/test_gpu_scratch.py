"""Scratch of the reduction, the back-transform and the residuals
(hsr_scratch.h): inside a stream capture it belongs to the graph, so replays
give the same after larger direct calls, after the capturing thread has ended
and beside direct calls on other streams."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(torch, n, ncols, graded, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((n, n))
    if graded:
        d = 10.0 ** (-12 * np.arange(n) / (n - 1))
        A *= d[:, None] * d
    return (torch.from_numpy(A).cuda(), torch.from_numpy(rng.standard_normal((ncols, n))).cuda(),
            torch.from_numpy(rng.uniform(-1, 1, ncols)).cuda())


def _all(hsr, torch, A0, X0, wr, stream=None):
    A, X = A0.clone(), X0.clone()
    tau = hsr.hessenberg_device(A, stream=stream)
    hsr.hessenberg_apply_q_device(A, tau, X, stream=stream)
    return A, tau, X, hsr.residuals_device(A0, wr, X0, stream=stream)


def _capture(hsr, torch, A0, X0, wr):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = _all(hsr, torch, A0, X0, wr, torch.cuda.current_stream())
    return g, out


def _same(torch, got, ref):
    for a, b in zip(got[:3], ref[:3]):
        assert torch.equal(a, b)
    torch.testing.assert_close(got[3], ref[3], rtol=1e-13, atol=0)     # sums by atomics: any order


@pytest.mark.parametrize("n,ncols,graded", [(20, 3, False), (200, 70, False), (200, 70, True), (2100, 40, False)])
def test_replay_after_larger_calls(gpu_lib, n, ncols, graded):
    import torch
    import hsrq3in_gb300 as hsr
    p = _problem(torch, n, ncols, graded, 1)
    ref = _all(hsr, torch, *p)
    torch.cuda.synchronize()
    g, out = _capture(hsr, torch, *p)
    big = _problem(torch, n + 500, ncols + 300, False, 2)
    for _ in range(2):
        _all(hsr, torch, *big)
        for t in out:
            t.zero_()
        g.replay()
        torch.cuda.synchronize()
        _same(torch, out, ref)


def test_first_call_in_a_capture(gpu_lib):
    """A thread without scratch captures, ends, and the graph is replayed."""
    import torch
    import hsrq3in_gb300 as hsr
    p = _problem(torch, 300, 40, False, 3)
    ref = _all(hsr, torch, *p)
    box = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            box.append(_capture(hsr, torch, *p))
    t = threading.Thread(target=work)
    t.start()
    t.join()
    g, out = box[0]
    for _ in range(2):
        for t in out:
            t.zero_()
        g.replay()
        torch.cuda.synchronize()
        _same(torch, out, ref)


def test_replay_beside_direct_calls(gpu_lib):
    import torch
    import hsrq3in_gb300 as hsr
    p, q = _problem(torch, 400, 60, False, 4), _problem(torch, 380, 50, False, 5)
    ref, qref = _all(hsr, torch, *p), _all(hsr, torch, *q)
    g, out = _capture(hsr, torch, *p)
    s = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.cuda.stream(s[0]):
            g.replay()
        with torch.cuda.stream(s[1]):
            direct = _all(hsr, torch, *q, s[1])
    torch.cuda.synchronize()
    _same(torch, out, ref)
    _same(torch, direct, qref)


def test_streams_that_come_and_go(gpu_lib):
    """One thread, each call on a stream of its own that is destroyed behind
    it with the work still enqueued, residuals included: a new stream may get a
    destroyed one's handle."""
    import ctypes
    import torch
    import hsrq3in_gb300 as hsr
    rt = ctypes.CDLL("libcudart.so." + torch.version.cuda.split(".")[0])
    probs = [_problem(torch, n, 90, False, n) for n in (600, 300, 500, 200, 60)]
    ref = [_all(hsr, torch, *p) for p in probs]
    torch.cuda.synchronize()

    class Stream:
        cuda_stream = None
    for _ in range(3):
        outs, copies = [], [(A0.clone(), X0.clone()) for A0, X0, _ in probs]
        torch.cuda.synchronize()
        for (A0, X0, wr), (A, X) in zip(probs, copies):
            s, h = Stream(), ctypes.c_void_p()
            assert rt.cudaStreamCreateWithFlags(ctypes.byref(h), 1) == 0
            s.cuda_stream = h.value
            tau = hsr.hessenberg_device(A, stream=s)
            hsr.hessenberg_apply_q_device(A, tau, X, stream=s)
            outs.append((A, tau, X, hsr.residuals_device(A0, wr, X0, stream=s)))
            assert rt.cudaStreamDestroy(h) == 0
        torch.cuda.synchronize()
        for got, r in zip(outs, ref):
            _same(torch, got, r)


def test_release_gives_everything_back(gpu_lib):
    """hsr_release_workspace frees the scratch of all three, which is no more
    than what their digits take (a triangle of V three times, n = 3000: 24
    blocks of 128 reflectors, 300 of their 128 x 128 blocks at 256 KB, 2 MB of
    Gram parts a block, and X;
    8 n^2 bytes for the reduction; H and X for the residuals), and later calls
    get it anew."""
    import torch
    import hsrq3in_gb300 as hsr
    n, ncols, mb = 3000, 64, 2.0 ** 20
    A0, X0, wr = _problem(torch, n, ncols, False, 6)
    A, X = A0.clone(), X0.clone()
    lib = hsr.load()
    _all(hsr, torch, A0, X0, wr)                                # library and allocator pools loaded
    lib.hsr_release_workspace()
    torch.cuda.synchronize()

    def used(f):
        before = torch.cuda.mem_get_info()[0]
        f()
        torch.cuda.synchronize()
        return (before - torch.cuda.mem_get_info()[0]) / mb
    tau = torch.zeros(n, dtype=torch.float64, device="cuda")
    res = torch.zeros(ncols, dtype=torch.float64, device="cuda")
    base = torch.cuda.mem_get_info()[0]
    red = used(lambda: lib.hsr_hessenberg_device(n, A.data_ptr(), n, tau.data_ptr(), None))
    back = used(lambda: lib.hsr_hessenberg_apply_q_device(n, A.data_ptr(), n, tau.data_ptr(), ncols, X.data_ptr(), n, None))
    val = used(lambda: lib.hsr_residuals_device(n, A0.data_ptr(), n, ncols, wr.data_ptr(), X0.data_ptr(), n, res.data_ptr(),
                                                None))
    assert 50 < red < 300 and 3 * 300 / 4 <= back < 3 * 300 / 4 + 80 and 100 < val < 200, (red, back, val)
    lib.hsr_release_workspace()
    assert base - torch.cuda.mem_get_info()[0] <= 8 * mb       # (the driver may keep a little)
    _same(torch, _all(hsr, torch, A0, X0, wr), (A, tau, X, res))
