"""log|det| of FP32 draws with a dense core of at most 128 nodes: the kernel that takes
four blocks per SM against the one it replaces there, which forecasts still take when
the iterative solve is switched off (the same operations, so the same factors: the
forecasts' log|det| of the same draws agree to the rounding of the FP64 sum of the
pivots' logarithms), at cores of one node, below, at and above each panel, and around
the largest; and draws that need pivoting.
"""
import numpy as np
import pytest

import oracle
from gpusgdlm_gb300 import SGDLM

pytestmark = pytest.mark.gpu


def _engine(m, kmax, seed, spread):
    import bench

    wl = bench.make_workload(m=m, kmax=kmax, T=2, seed=seed)
    P = wl["P"]
    s = SGDLM(1, strict=True)
    s.setSimultaneousParents(wl["p"], np.where(wl["sp"] >= m * m, np.nan, wl["sp"]).astype(float))
    s.setDiscountFactors(np.full(m, 0.97), np.full((P, P, m), 0.98))
    rng = np.random.default_rng(seed)
    par = (rng.uniform(-spread, spread, size=(P, m)),
           np.repeat((1e-6 * np.eye(P))[:, :, None], m, axis=2), np.full(m, 50.0), np.full(m, 1.0))
    return s, wl, par


def _both(s, wl, par, n, seed):
    s.setPosteriorParameters(*par)
    s.setRngState(seed, 0)
    s.computeVBPosterior(n, n)
    flags = s.getStats()["draws_pivoted"]
    d = s.getDraws()
    s.setPriorParameters(*par)
    s.setForecastSolver(False)
    s.setRngState(seed, 0)
    s.computeForecast(n, n, np.zeros((wl["P"], wl["m"])))
    f = s.getDraws()
    np.testing.assert_array_equal(d["thetas"], f["thetas"])
    return d, f, flags


@pytest.mark.parametrize("m,kmax,n", [
    (33, 1, 3), (40, 9, 700), (60, 17, 300), (90, 12, 1300), (120, 9, 200), (150, 12, 333),
    (170, 12, 200), (180, 13, 150), (200, 13, 100), (210, 13, 100), (240, 17, 300),
    (255, 17, 100), (275, 17, 60)])
def test_matches_the_large_kernel(built_lib, m, kmax, n):
    s, wl, par = _engine(m, kmax, 3 + m, min(0.3, 0.8 / kmax))
    d, f, flags = _both(s, wl, par, n, 5)
    assert flags == 0
    np.testing.assert_allclose(d["log_dets"], f["log_dets"], rtol=0, atol=1e-12)
    ld = oracle.logdet(wl["sp"], np.asfortranarray(d["thetas"][:, :, :16].transpose(0, 2, 1)))
    np.testing.assert_allclose(d["log_dets"][:16], ld, rtol=0, atol=1e-4)
    s.close()


def test_cores_cover_the_panels(built_lib):
    """The sizes above reach every panel count of the kernel and the first one beyond."""
    cores = set()
    for m, kmax in ((33, 1), (90, 12), (120, 9), (150, 12), (180, 13), (210, 13), (275, 17)):
        s, _, _ = _engine(m, kmax, 3 + m, 0.1)
        cores.add((s.getEliminationInfo()["core_n"] + 31) // 32)
        s.close()
    assert {1, 2, 3, 4, 5} <= cores


def test_draws_that_need_pivoting(built_lib):
    s, wl, par = _engine(100, 10, 8, 3.0)
    s.setPosteriorParameters(*par)
    s.computeVBPosterior(64, 64)
    assert s.getStats()["draws_pivoted"] > 0
    d = s.getDraws()
    ld = oracle.logdet(wl["sp"], np.asfortranarray(d["thetas"].transpose(0, 2, 1)))
    # partial pivoting in FP32: growth and condition of these draws (spectral radius far
    # above one) leave about four digits
    np.testing.assert_allclose(d["log_dets"], ld, rtol=0, atol=5e-2)
    s.close()


@pytest.mark.parametrize("m,kmax,n", [(275, 17, 305), (290, 17, 700), (345, 17, 400), (400, 17, 611)])
def test_last_rows_by_the_small_kernel(built_lib, m, kmax, n):
    """Cores of 160, 192 and 224 rows with more draws than the large kernel has blocks: it
    leaves their last 128 rows to the small one."""
    s, wl, par = _engine(m, kmax, 3 + m, min(0.3, 0.8 / kmax))
    assert 128 < s.getEliminationInfo()["core_n"] <= 224
    d, f, flags = _both(s, wl, par, n, 5)
    assert flags == 0
    np.testing.assert_allclose(d["log_dets"], f["log_dets"], rtol=0, atol=1e-12)
    s.close()


@pytest.mark.parametrize("m,spread", [(275, 1.0), (275, 3.0), (345, 3.0)])
def test_last_rows_of_draws_that_need_pivoting(built_lib, m, spread):
    """A check that fails before or in the last 128 rows sends the draw to the redo: the
    first of many draws (two kernels) against the same draws alone (one kernel), whose
    operations are the same up to the FP64 sum of the logarithms."""
    s, wl, par = _engine(m, 17, 3 + m, spread)
    got = []
    for n in (200, 330):
        s.setPosteriorParameters(*par)
        s.setRngState(5, 0)
        s.computeVBPosterior(n, n)
        got.append((s.getStats()["draws_pivoted"], s.getDraws()))
    (few_flags, few), (many_flags, many) = got
    np.testing.assert_array_equal(few["thetas"], many["thetas"][..., :200])
    np.testing.assert_allclose(few["log_dets"], many["log_dets"][:200], rtol=0, atol=1e-10)
    assert few_flags <= many_flags <= few_flags + 130
    assert spread < 3.0 or few_flags > 0
    s.close()


def test_last_rows_in_two_parts(built_lib):
    """More draws than one hand-over takes (16 384): the first draws against the same draws
    alone, and the second part's log weights against the first's (independent draws of one
    distribution: means within six standard errors, standard deviations within a tenth)."""
    s, wl, par = _engine(275, 17, 278, 0.05)
    logw = []
    for n in (250, 16500):
        s.setPosteriorParameters(*par)
        s.setRngState(5, 0)
        w = s.computeVBPosterior(n, n)["IS_weights"]
        assert s.getStats()["draws_pivoted"] == 0
        assert np.all(w > 0) and abs(w.sum() - 1.0) < 1e-12
        logw.append(np.log(w))
    few, many = logw
    np.testing.assert_allclose(many[:250] - many[0], few - few[0], rtol=0, atol=1e-10)
    a, b = many[:8250], many[8250:]
    assert abs(a.mean() - b.mean()) <= 6 * many.std() * np.sqrt(2 / 8250)
    assert abs(a.std() - b.std()) <= 0.1 * many.std()
    s.close()
