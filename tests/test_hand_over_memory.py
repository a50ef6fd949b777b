"""Memory of the hand-over between the two kernels of FP32 log|det| (cores of 160 to 224
rows): a buffer of its own only while most of the device's memory is free, else the room
behind the Gamma copy, else one kernel; the values are the same (one kernel adds the FP64
logarithms in another order: 1e-12, as test_small_core.py), and no size is refused for
the lack of it."""
import contextlib

import numpy as np
import pytest
import torch

from gpusgdlm_gb300 import SGDLM, Batch
from gpusgdlm_gb300.sgdlm import _pd

pytestmark = pytest.mark.gpu

SIM_NOT_INIT, OUT_OF_MEMORY = 4, 8  # status codes of include/sgdlm.h
M, KMAX, SLAB = 275, 17, 4 * (128 * 128 + 32)


def _engine():
    import bench

    wl = bench.make_workload(m=M, kmax=KMAX, T=2, seed=278)
    s = SGDLM(1, strict=True)
    s.setSimultaneousParents(wl["p"], np.where(wl["sp"] >= M * M, np.nan, wl["sp"]).astype(float))
    P = wl["P"]
    s.setDiscountFactors(np.full(M, 0.97), np.full((P, P, M), 0.98))
    assert 128 < s.getEliminationInfo()["core_n"] <= 224
    return s, wl


def _log_dets(s, wl, n):
    """log|det| of n draws and the launches of the call that made them."""
    P = wl["P"]
    rng = np.random.default_rng(1)
    s.setPosteriorParameters(rng.uniform(-0.05, 0.05, (P, M)),
                             np.repeat((1e-4 * np.eye(P))[:, :, None], M, axis=2), np.full(M, 50.0),
                             np.ones(M))
    s.setRngState(5, 0)
    assert s._lib.sgdlm_init_sim_memory(s._h, n, n) == 0
    before = s.launchCount()
    s.computeVBPosterior(n, n)
    launches = s.launchCount() - before
    ld = np.zeros(n)
    assert s._lib.sgdlm_get_draws(s._h, None, None, _pd(ld)) == 0
    assert s.getStats()["draws_pivoted"] == 0
    return ld, launches


@pytest.fixture(autouse=True)
def _free_device():
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < _most() + (4 << 30):
        pytest.skip("another process holds the device's memory")


@contextlib.contextmanager
def _hold(keep_free):
    """The device's free memory but keep_free bytes, for a while."""
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - keep_free, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def _most():
    return torch.cuda.mem_get_info()[1] // 8 * 7


@pytest.mark.parametrize("n,parts", [(2000, 0), (7000, 6)])
def test_little_free_memory(built_lib, n, parts):
    torch.cuda.empty_cache()
    s, wl = _engine()
    ld, launches = _log_dets(s, wl, n)  # (a kernel pair of one part)
    s.close()
    with _hold(_most()):
        s, _ = _engine()
        got, now = _log_dets(s, wl, n)
        s.close()
    if parts:  # room for a share of the draws behind the Gamma copy
        room = n * (M * wl["P"] - int((wl["sp"] < M * M).sum())) * 4 // SLAB
        assert 4 * 304 <= room and -(-n // room) == parts
        assert now == launches + 2 * (parts - 1)
        np.testing.assert_array_equal(got, ld)
    else:
        assert now == launches - 1
        np.testing.assert_allclose(got, ld, rtol=0, atol=1e-12)


def test_no_size_is_refused_for_it(built_lib):
    """The memory that is left holds the engine, but not its hand-over buffer."""
    n = 7000
    torch.cuda.empty_cache()
    s, wl = _engine()
    ld, _ = _log_dets(s, wl, n)
    s.close()
    with _hold(_most()):
        free0 = torch.cuda.mem_get_info()[0]
        s, _ = _engine()
        got, _ = _log_dets(s, wl, n)
        need = free0 - torch.cuda.mem_get_info()[0]
        s.close()
    with _hold(need + n * SLAB // 2):
        s, _ = _engine()
        tight, _ = _log_dets(s, wl, n)
        s.close()
    np.testing.assert_array_equal(got, ld)
    np.testing.assert_array_equal(tight, ld)


def test_the_buffer_goes_first(built_lib):
    """An engine that grows gives its hand-over buffer up rather than fail."""
    small, large = 3000, 7000
    free = []
    with _hold(_most()):
        s, wl = _engine()
        for n in (small, large):  # without the buffer
            want, _ = _log_dets(s, wl, n)
            free.append(torch.cuda.mem_get_info()[0])
        s.close()
    s, _ = _engine()
    _log_dets(s, wl, small)
    with _hold(free[0] - free[1] - small * SLAB // 2):
        got, _ = _log_dets(s, wl, large)
        s.close()
    np.testing.assert_array_equal(got, want)


def test_recorded_steps_keep_their_buffers(built_lib):
    """A batch's recorded step stays valid while the draw count goes up and down within what
    the engine has held before (here in FP64, which has no hand-over)."""
    P = _engine()[1]["P"]
    n, out = 1000, []
    for detour in (False, True):
        s, wl = _engine()
        s.setPrecision("fp64")
        assert s._lib.sgdlm_init_sim_memory(s._h, 3000, 3000) == 0
        s.setPrecision("mixed")
        assert s._lib.sgdlm_init_sim_memory(s._h, n, n) == 0
        s.setPriorParameters(np.zeros((P, M)), np.repeat((1e-3 * np.eye(P))[:, :, None], M, axis=2),
                             np.full(M, 50.0), np.ones(M))
        s.setRngState(5, 0)
        y, F, x = (torch.from_numpy(np.ravel(v, order="F").copy()).cuda()
                   for v in (wl["y"][1], wl["F_of"](1), wl["F_of"](2, False)))
        w, fc = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (n, n * M))
        torch.cuda.synchronize()
        b = Batch([s])
        b.record([y.data_ptr()], [F.data_ptr()], [x.data_ptr()], 0.0, [fc.data_ptr()], [w.data_ptr()])
        if detour:
            for k in (2500, n):
                assert s._lib.sgdlm_init_sim_memory(s._h, k, k) == 0
        b.step()
        s.synchronize()
        out.append((w.cpu().numpy(), fc.cpu().numpy()))
        b.close()
        s.close()
    assert np.all(out[0][0] > 0) and np.isfinite(out[0][1]).all()
    for a, c in zip(*out):
        np.testing.assert_array_equal(a, c)


def test_plan_without_memory(built_lib):
    """A plan whose scratch cannot be had gives the simulation memory back; with memory it
    is set up anew."""
    n = 310
    s, wl = _engine()
    want, _ = _log_dets(s, wl, n)
    with _hold(8 << 20):  # (no levels: 288 x 288 values per block, 100 MB)
        assert s._lib.sgdlm_set_elimination_levels(s._h, 0) == OUT_OF_MEMORY
        assert s.nsim == 0
        assert s._lib.sgdlm_compute_vb_posterior(s._h, None, None, None, None, None, None) == SIM_NOT_INIT
    got, _ = _log_dets(s, wl, n)
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-4)  # another elimination order
    s.close()
