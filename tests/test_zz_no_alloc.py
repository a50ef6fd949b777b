"""The allocation-free log|det| entry point (sgdlm_log_det_noalloc).

It serves callers that must not allocate device memory; its LU working
matrices live in a static device array.  Checked here against the FP64 oracle's
log|det| of the same FP32 draws (and against the regular, allocating entry
point's), on two calls in a row, since the static array keeps the previous
call's contents.  This file runs last so that a failure here comes after every
other test has run.

Tolerance: the oracle runs a partial-pivoting LU in FP64 on the very FP32
values the GPU read, so the difference is the FP32 factorisation's own
rounding.  This entry point factors the whole matrix densely (no sparse
levels); with these draws (coefficients 0.05 +- 0.045, row sums up to 0.85) that
rounding reaches 2.4e-5 in log|det|, hence 5e-5 here.  Against the allocating
entry point (the same kernels on the same draws) the results agree to 1e-9.
"""
import ctypes

import numpy as np
import pytest

import oracle
from gpusgdlm_gb300 import SGDLM
from gpusgdlm_gb300 import _lib as L

LOGDET_ATOL = 5e-5

pytestmark = pytest.mark.gpu


def _engine_draws(m, P, p, sp, mt, C, n, precision="mixed", seed=17):
    s = SGDLM(1, strict=True, precision=precision)
    s.setSimultaneousParents(p, sp)
    s.setWarpLu(False)  # the block LU kernels at every m, as the no-alloc path runs
    s.setEliminationLevels(0)  # the dense LU of the whole matrix, as the no-alloc path runs
    s.setDiscountFactors(np.full(m, 0.95), np.full((P, P, m), 0.95))
    s.setPosteriorParameters(mt, C, np.full(m, 20.0), np.full(m, 0.01))
    s.setRngState(seed, 0)
    s.computeVBPosterior(n, n)
    d = s.getDraws()
    st = s.getStats()
    s.close()
    return d, st


def _call_noalloc(m, P, n, theta_sm, sp_u32):
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda:0")
    th = torch.tensor(theta_sm, dtype=torch.float32, device=dev)
    sp = torch.tensor(sp_u32.view(np.int32).ravel(order="F"), dtype=torch.int32, device=dev)
    outs = []
    for _ in range(2):
        ld = torch.full((n,), np.nan, dtype=torch.float64, device=dev)
        fl = torch.full((n,), -1, dtype=torch.int32, device=dev)
        st = L.lib().sgdlm_log_det_noalloc(m, P, n, ctypes.c_void_p(th.data_ptr()),
                                           ctypes.c_void_p(sp.data_ptr()),
                                           ctypes.c_void_p(ld.data_ptr()),
                                           ctypes.c_void_p(fl.data_ptr()), None)
        assert st == 0
        torch.cuda.synchronize()
        outs.append((ld.cpu().numpy(), fl.cpu().numpy()))
    return outs


def _series_major(thetas_ref_layout):
    # (max_p, m, n) reference layout -> (m, n, max_p) series-major, FP32 exact
    return np.ascontiguousarray(thetas_ref_layout.transpose(1, 2, 0)).astype(np.float32)


def _oracle_logdet(sp_u32, theta_sm_f32):
    # series-major FP32 (m, n, P) -> the oracle's (P, n, m) FP64 layout, same values
    th = np.asfortranarray(theta_sm_f32.astype(np.float64).transpose(2, 1, 0))
    return oracle.logdet(sp_u32, th)


def test_noalloc_matches_oracle_m400():
    import bench

    wl = bench.make_workload(m=400, T=3, seed=5)
    m, P, n = wl["m"], wl["P"], 700
    sp = np.where(wl["sp"] >= m * m, np.nan, wl["sp"]).astype(float)
    mt = np.full((P, m), 0.05)
    C = np.repeat((0.002 * np.eye(P))[:, :, None], m, axis=2)
    d, _ = _engine_draws(m, P, wl["p"], sp, mt, C, n)
    th = _series_major(d["thetas"])
    ref = _oracle_logdet(wl["sp"], th)
    for ld, fl in _call_noalloc(m, P, n, th, wl["sp"]):
        err = np.abs(ld - ref)
        print(f"m=400 no-alloc log|det| max abs error vs oracle {err.max():.3e}")
        np.testing.assert_allclose(ld, ref, rtol=0, atol=LOGDET_ATOL)
        np.testing.assert_allclose(ld, d["log_dets"], rtol=0, atol=1e-9)
        assert np.all(fl >= 0)


@pytest.mark.parametrize("m,kmax,n", [(225, 6, 70), (256, 5, 1), (257, 9, 130), (333, 11, 67), (460, 4, 40),
                                      (736, 3, 10)])
def test_noalloc_several_blocks_per_draw(m, kmax, n):
    """Matrices of which the 16 MiB array holds fewer than the GPU has SMs: a cluster of
    blocks shares each draw (column shares of every width, one draw, more draws than
    matrices).  The same operations as the allocating entry point's dense LU."""
    import bench

    wl = bench.make_workload(m=m, kmax=kmax, T=3, seed=m)
    P = wl["P"]
    sp = np.where(wl["sp"] >= m * m, np.nan, wl["sp"]).astype(float)
    d, st = _engine_draws(m, P, wl["p"], sp, np.full((P, m), 0.05), np.repeat((0.001 * np.eye(P))[:, :, None], m, axis=2), n)
    th = _series_major(d["thetas"])
    for ld, fl in _call_noalloc(m, P, n, th, wl["sp"]):
        np.testing.assert_allclose(ld, d["log_dets"], rtol=0, atol=1e-9)
        assert (np.asarray(fl) != 0).sum() == st["draws_pivoted"]


def test_noalloc_matches_oracle_with_pivoting():
    m, P, n = 3, 1, 300
    sp = np.array([[0 + 3 * 1, 1 + 3 * 0, 2 + 3 * 0]], dtype=np.float64)
    mt = np.array([[0.3, 20.0, -15.0]])
    C = np.full((1, 1, m), 1e-4)
    d, st = _engine_draws(m, P, [1, 1, 1], sp, mt, C, n)
    assert st["draws_pivoted"] == n
    th = _series_major(d["thetas"])
    ref = _oracle_logdet(sp.astype(np.uint32), th)
    for ld, fl in _call_noalloc(m, P, n, th, sp.astype(np.uint32)):
        np.testing.assert_allclose(ld, ref, rtol=0, atol=LOGDET_ATOL)
        assert np.all(fl & 8)  # every draw went through the pivoting redo


@pytest.mark.parametrize("m", [737, 1000, 2048, 3000])
def test_noalloc_rejects_m_above_its_limit(m):
    """736 series is the largest m whose LU block fits the shared memory of one
    block; every larger m is refused before any pointer is used."""
    dummy = ctypes.c_void_p(16)  # never dereferenced: the size check comes first
    st = L.lib().sgdlm_log_det_noalloc(m, 4, 10, dummy, dummy, dummy, dummy, None)
    assert st == 9  # SGDLM_ERR_UNSUPPORTED
