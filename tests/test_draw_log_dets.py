"""log|det| of a forecast's FP64 draws, which the iterative solve does not need and
getDraws computes: what is called in between must not change them.

Tolerance: as in test_forecast_iterative.py, 1e-12 for draws with small multipliers;
draws that need pivoting (multipliers above the limit in most of them) 1e-8, as in
test_logdet64.py.
"""
import numpy as np
import pytest
import torch

import oracle
from gpusgdlm_gb300 import SGDLM, Batch
from gpusgdlm_gb300.sgdlm import _pd

pytestmark = pytest.mark.gpu


def _engine(m, kmax, seed=3, spread=0.05, full=False, levels=None):
    """full: every series has kmax parents and one other coefficient."""
    import bench

    if full:
        rng = np.random.default_rng(seed)
        sp = np.full((kmax + 1, m), 2147483648, dtype=np.uint32, order="F")
        for j in range(m):
            sp[1:, j] = j + m * rng.choice(np.delete(np.arange(m), j), size=kmax, replace=False)
        wl = dict(P=kmax + 1, p=np.full(m, kmax + 1), sp=sp, x=rng.normal(0, 1, (kmax + 1, m)))
    else:
        wl = bench.make_workload(m=m, kmax=kmax, T=4, seed=seed)
        wl["x"] = wl["F_of"](2, False)
    P = wl["P"]
    s = SGDLM(1, strict=True, precision="fp64")
    s.setCompat(0)  # the reference's beta sampler gives NaN for some of these shapes
    s.setSimultaneousParents(wl["p"], _sp(wl["sp"], m))
    if levels is not None:
        s.setEliminationLevels(levels)
    s.setDiscountFactors(np.full(m, 0.97), np.full((P, P, m), 0.98))
    rng = np.random.default_rng(seed)
    s.setPosteriorParameters(rng.uniform(-spread, spread, size=(P, m)),
                             np.repeat((0.04 * spread**2 * np.eye(P))[:, :, None], m, axis=2),
                             np.full(m, 20.0), np.full(m, 1.0))
    s.computePrior()
    s.setRngState(11, 0)
    return s, wl


def _sp(sp, m):
    return np.where(sp >= m * m, np.nan, sp).astype(float)


def _thetas(s):
    m, P, n = s.m, s.max_p, s.nsim
    th = np.zeros((P, m, n), order="F")
    assert s._lib.sgdlm_get_draws(s._h, None, _pd(th), None) == 0
    return np.asfortranarray(th.transpose(0, 2, 1))


def _log_dets(s):
    ld = np.zeros(s.nsim)
    assert s._lib.sgdlm_get_draws(s._h, None, None, _pd(ld)) == 0
    return ld


@pytest.mark.parametrize("m,kmax,spread,tol", [(70, 6, 0.05, 1e-12), (100, 10, 3.0, 1e-8)])
def test_other_parents(built_lib, m, kmax, spread, tol):
    s, wl = _engine(m, kmax, spread=spread)
    s.computeForecast(200, 200, wl["x"])
    ld = oracle.logdet(wl["sp"], _thetas(s))
    # the same series, every simultaneous parent another one
    import bench

    other = bench.make_workload(m=m, kmax=kmax, T=2, seed=77)
    assert other["P"] == wl["P"] and not np.array_equal(other["sp"], wl["sp"])
    s.setSimultaneousParents(other["p"], _sp(other["sp"], m))
    np.testing.assert_allclose(_log_dets(s), ld, rtol=0, atol=tol)
    s.close()


# room for the old draws' Gamma entries beside the new ones, none, no levels, and draws
# pivoted in the core (3) and over the whole matrix (1e6: multipliers beyond the levels' limit)
@pytest.mark.parametrize("m,kmax,full,levels,spread,tol", [
    (70, 6, False, None, 0.05, 1e-12), (70, 10, True, None, 0.02, 1e-12), (70, 6, False, 0, 0.05, 1e-12),
    (100, 10, False, None, 3.0, 1e-8), (100, 10, False, None, 1e6, 1e-8)])
def test_evolved_draws(built_lib, m, kmax, full, levels, spread, tol):
    s, wl = _engine(m, kmax, spread=spread, full=full, levels=levels)
    s.computeForecast(200, 200, wl["x"])
    ld = oracle.logdet(wl["sp"], _thetas(s))
    before = _thetas(s)
    assert s._lib.sgdlm_init_forecast_priors(s._h) == 0
    for _ in range(2):
        assert s._lib.sgdlm_evolve_forecast_samples(s._h) == 0
    assert np.abs(_thetas(s) - before).max() > 0
    np.testing.assert_allclose(_log_dets(s), ld, rtol=0, atol=tol)
    # and a forecast of the evolved draws replaces them
    s.computeForecast(200, 200, np.stack([wl["x"]] * 2, axis=2))
    np.testing.assert_allclose(_log_dets(s), oracle.logdet(wl["sp"], _thetas(s)), rtol=0, atol=tol)
    s.close()


def test_another_precision_or_plan(built_lib):
    s, wl = _engine(70, 6)
    s.computeForecast(200, 200, wl["x"])
    ld = oracle.logdet(wl["sp"], _thetas(s))
    s.setEliminationLevels(0)
    s.setPrecision("mixed")
    np.testing.assert_allclose(_log_dets(s), ld, rtol=0, atol=1e-12)
    s.close()


def test_recorded_step_not_run(built_lib):
    """Recording a batch's step draws nothing: the log|det| stay those of the forecast."""
    s, wl = _engine(70, 6)
    m, P = s.m, s.max_p
    s.computeForecast(200, 200, wl["x"])
    ld = oracle.logdet(wl["sp"], _thetas(s))
    y, F = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (m, P * m))
    b = Batch([s])
    b.record([y.data_ptr()], [F.data_ptr()])
    np.testing.assert_allclose(_log_dets(s), ld, rtol=0, atol=1e-12)
    b.close()
    s.close()


def test_memory_given_back(built_lib):
    """Nothing is computed from draws that are gone."""
    s, wl = _engine(70, 6)
    s.computeForecast(200, 200, wl["x"])
    assert s._lib.sgdlm_clear_sim_memory(s._h) == 0
    s.setPrecision("mixed")
    s.setSimultaneousParents(wl["p"], np.full((s.max_p, s.m), np.nan))
    s.close()
