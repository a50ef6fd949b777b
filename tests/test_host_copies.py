"""The staged copies between the caller's arrays and the device: several threads on one
handle, device memory in the place of the arrays, and every size around the limits of
what is staged."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from gpusgdlm_gb300 import SGDLM

pytestmark = pytest.mark.gpu


def _engine(m, kmax=4, n_ext=3, seed=2):
    import bench

    wl = bench.make_workload(m=m, kmax=kmax, n_ext=n_ext, T=4, seed=seed)
    P = wl["P"]
    s = SGDLM(1, strict=True)
    s.setSimultaneousParents(wl["p"], np.where(wl["sp"] >= m * m, np.nan, wl["sp"]).astype(float))
    s.setDiscountFactors(np.full(m, 0.97), np.full((P, P, m), 0.98))
    rng = np.random.default_rng(seed)
    par = (rng.uniform(-0.05, 0.05, size=(P, m)), np.repeat((1e-4 * np.eye(P))[:, :, None], m, axis=2),
           np.full(m, 20.0), np.full(m, 1.0))
    return s, wl, par


def test_results_while_another_thread_asks(built_lib):
    """Reading sizes, statistics and parameters beside a running call changes nothing
    of either's results."""
    s, wl, par = _engine(20)
    y, F = wl["y"][2], wl["F_of"](2)
    s.setPriorParameters(*par)
    s.computePosterior(y, F)
    post = s.getParameters()
    s.setRngState(5, 0)
    vb = s.computeVBPosterior(300, 300)
    stop, wrong, asked = threading.Event(), [], [0]

    def ask():
        while not stop.is_set():
            asked[0] += 1
            if (s.m, s.max_p, s.nsim) != (20, wl["P"], 300) or s.getStats()["ess"] < 0:
                wrong.append("sizes")
            if not np.array_equal(s.getDiscountFactors()["beta"], np.full(20, 0.97)):
                wrong.append("discount factors")

    t = threading.Thread(target=ask)
    t.start()
    try:
        for _ in range(200):
            s.setPriorParameters(*par)
            s.computePosterior(y, F)
            got = s.getParameters()
            for k in post:
                np.testing.assert_array_equal(got[k], post[k])
            s.setRngState(5, 0)
            again = s.computeVBPosterior(300, 300)
            for k in ("m", "C", "n", "s", "IS_weights"):
                np.testing.assert_array_equal(again[k], vb[k])
    finally:
        stop.set()
        t.join()
    assert not wrong and asked[0] > 0
    s.close()


def test_arrays_in_device_memory(built_lib):
    """A copy's direction is its addresses': arrays in device memory are served, large
    and small, as host arrays."""
    s, wl, par = _engine(40)
    P, m, n = s.max_p, s.m, 2000  # (n m doubles are beyond what is staged)
    s.setPriorParameters(*par)
    s.setRngState(3, 0)
    x = np.asfortranarray(wl["F_of"](2, False))
    ref = s.computeForecast(n, n, x)
    want = s.getParameters()

    def on_gpu(a):
        return torch.from_numpy(np.ravel(np.asarray(a, dtype=np.float64), order="F").copy()).cuda()

    def ptr(t):
        return C.cast(t.data_ptr(), C.POINTER(C.c_double))

    d = [on_gpu(par[0] + 1), on_gpu(par[1]), on_gpu(par[2]), on_gpu(par[3])]
    torch.cuda.synchronize()
    assert s._lib.sgdlm_set_parameters(s._h, *[ptr(t) for t in d]) == 0
    np.testing.assert_array_equal(s.getParameters()["m"], par[0] + 1)
    s.setPriorParameters(*par)
    assert s._lib.sgdlm_get_parameters(s._h, *[ptr(t) for t in d]) == 0
    for t, k in zip(d, ("m", "C", "n", "s")):
        np.testing.assert_array_equal(t.cpu().numpy(), np.ravel(want[k], order="F"))
    s.setRngState(3, 0)
    out, dx = torch.zeros(n * m, dtype=torch.float64, device="cuda"), on_gpu(x)
    torch.cuda.synchronize()
    assert s._lib.sgdlm_compute_forecast(s._h, ptr(out), ptr(dx), None, None, 0) == 0
    np.testing.assert_array_equal(out.cpu().numpy(), np.ravel(ref, order="F"))
    s.close()


# P*P*m doubles beside 128 KiB (16 384), and beyond 1 MiB in all
@pytest.mark.parametrize("m", [1, 334, 335, 1700])
def test_sizes_around_the_stage(built_lib, m):
    s, wl, _ = _engine(m, kmax=min(4, m - 1))
    P = s.max_p
    rng = np.random.default_rng(m)
    A, b = rng.normal(size=(P, P, m)), rng.normal(size=m)
    s.setDiscountFactors(b, A)
    s.setPriorParameters(rng.normal(size=(P, m)), A + 1, b + 2, b + 3)
    got, par = s.getDiscountFactors(), s.getParameters()
    np.testing.assert_array_equal(got["beta"], b)
    np.testing.assert_array_equal(got["delta"], A)
    np.testing.assert_array_equal(par["C"], A + 1)
    np.testing.assert_array_equal(par["n"], b + 2)
    np.testing.assert_array_equal(par["s"], b + 3)
    s.close()
