"""Evolution of draws whose state noise is not finite: theta + U_W' omega is a sum over all
max_p coefficients, so that a NaN omega reaches the inactive ones too (as 0 times NaN), and
no other series."""
import numpy as np
import pytest

from gpusgdlm_gb300 import SGDLM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m,kmax", [(20, 4), (40, 5), (40, 9)])  # max_p 7, 8 and 12
def test_noise_that_is_not_finite(built_lib, precision, m, kmax):
    import bench

    wl = bench.make_workload(m=m, kmax=kmax, T=2, seed=6)
    P, p, bad = wl["P"], wl["p"], int(np.argmin(wl["p"]))
    assert p[bad] < P
    s = SGDLM(1, strict=True, precision=precision)
    s.setCompat(0)
    s.setSimultaneousParents(p, np.where(wl["sp"] >= m * m, np.nan, wl["sp"]).astype(float))
    s.setDiscountFactors(np.full(m, 0.97), np.full((P, P, m), 0.98))
    par = (np.full((P, m), 0.01), np.repeat((1e-4 * np.eye(P))[:, :, None], m, axis=2),
           np.full(m, 20.0), np.ones(m))
    s.setPosteriorParameters(*par)
    s.computePrior()
    n = 300
    s.computeForecast(n, n, np.zeros((P, m)))
    before = s.getDraws()["thetas"]
    assert np.isfinite(before).all()
    c = np.ones(m)
    c[bad] = np.nan
    s.setPriorParameters(*par[:3], c)
    assert s._lib.sgdlm_init_forecast_priors(s._h) == 0
    assert s._lib.sgdlm_evolve_forecast_samples(s._h) == 0
    after = s.getDraws()["thetas"]
    assert np.isnan(after[:, bad, :]).all()
    others = np.arange(m) != bad
    assert np.isfinite(after[:, others, :]).all()
    for j in np.flatnonzero(others):  # inactive coefficients do not move
        np.testing.assert_array_equal(after[p[j]:, j, :], before[p[j]:, j, :])
    s.close()
