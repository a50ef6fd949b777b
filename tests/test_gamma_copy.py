"""The draw-major copy of the Gamma entries under parental sets that it was not written
for: coefficients of a series that address another row of (I - Gamma) (sp holds any
position row + m col), and draws kept while the sets change.  Against the oracle, at
sizes of every kernel that reads the copy.

Tolerance: FP64 1e-11 (as test_logdet64.py) and 1e-10 of a draw's largest forecast;
FP32 draws 1e-4 in log|det| (as test_small_core.py) and 1e-5 of a draw's largest
forecast (as test_gpu_parity.py).
"""
import numpy as np
import pytest

import oracle
from gpusgdlm_gb300 import SGDLM
from gpusgdlm_gb300.sgdlm import _pd

pytestmark = pytest.mark.gpu

NONE = 2147483648
TOL = {"fp64": (1e-11, 1e-10), "mixed": (1e-4, 1e-5)}


def _structure(m, kmax, seed, own_rows):
    """Up to kmax coefficients per series at distinct off-diagonal positions, the others
    external."""
    rng = np.random.default_rng(seed)
    P = kmax + 2
    sp = np.full((P, m), NONE, dtype=np.uint32, order="F")
    if own_rows:
        for j in range(m):
            q = rng.choice(np.delete(np.arange(m), j), size=rng.integers(0, kmax + 1), replace=False)
            sp[2:2 + len(q), j] = j + m * q
    else:  # the same number of entries anywhere
        pos = np.array([r + m * c for r in range(m) for c in range(m) if r != c])
        pos = rng.permutation(pos)[:m * kmax].reshape(kmax, m)
        sp[2:, :] = np.where(rng.random((kmax, m)) < 0.7, pos, NONE)
    return np.full(m, P), sp


def _set(s, p, sp):
    m = sp.shape[1]
    s.setSimultaneousParents(p, np.where(sp >= m * m, np.nan, sp).astype(float))


def _engine(m, kmax, precision, own_rows, seed=4):
    p, sp = _structure(m, kmax, seed, own_rows)
    P = sp.shape[0]
    s = SGDLM(1, strict=True, precision=precision)
    s.setCompat(0)
    _set(s, p, sp)
    s.setDiscountFactors(np.full(m, 0.97), np.full((P, P, m), 0.98))
    rng = np.random.default_rng(seed)
    par = (rng.uniform(-0.1, 0.1, size=(P, m)), np.repeat((1e-4 * np.eye(P))[:, :, None], m, axis=2),
           np.full(m, 20.0), np.full(m, 1.0))
    x = np.asfortranarray(rng.normal(0, 1, (P, m)))
    return s, sp, par, x


def _check_forecast(out_y, sp, d, x, seed, epoch, tol):
    lam = np.asfortranarray(d["lambdas"].T)
    th = np.asfortranarray(d["thetas"].transpose(0, 2, 1))
    y, _ = oracle.forecast(sp, lam, th, x, seed, epoch)
    assert (np.abs(out_y - y).max(axis=0) / np.abs(y).max(axis=0)).max() <= tol


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m,kmax,n", [(3, 1, 40), (6, 2, 200), (20, 4, 100), (45, 5, 300), (150, 8, 64),
                                      (290, 17, 330)])
def test_coefficients_of_other_rows(built_lib, precision, m, kmax, n):
    ld_tol, y_tol = TOL[precision]
    s, sp, par, x = _engine(m, kmax, precision, own_rows=False)
    s.setPosteriorParameters(*par)
    s.setRngState(5, 0)
    s.computeVBPosterior(n, n)
    d = s.getDraws()
    th = np.asfortranarray(d["thetas"].transpose(0, 2, 1))
    np.testing.assert_allclose(d["log_dets"], oracle.logdet(sp, th), rtol=0, atol=ld_tol)
    s.computePrior()
    s.setRngState(6, 0)
    for iterative in (True, False):
        s.setForecastSolver(iterative)
        s.setRngState(6, 0)
        _check_forecast(s.computeForecast(n, n, x), sp, s.getDraws(), x, 6, 0, y_tol)
    # evolved draws (the second step's; the sampler's epochs are 0, 1 and 2)
    s.setForecastSolver(True)
    s.setRngState(6, 0)
    y = s.computeForecast(n, n, np.stack([x, x], axis=2))
    _check_forecast(y[:, :, 1], sp, s.getDraws(), x, 6, 2, y_tol)
    s.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m,kmax,n", [(6, 2, 200), (20, 4, 100), (45, 5, 300), (290, 17, 330)])
@pytest.mark.parametrize("own_rows", [True, False])
def test_kept_draws_under_new_parents(built_lib, precision, m, kmax, n, own_rows):
    _, y_tol = TOL[precision]
    s, _, par, x = _engine(m, kmax, precision, own_rows=True)
    s.setPriorParameters(*par)
    s.setRngState(7, 0)
    s.computeForecast(n, n, x)
    p, sp = _structure(m, kmax, 99, own_rows)
    _set(s, p, sp)
    y = np.zeros((m, n), order="F")
    assert s._lib.sgdlm_compute_forecast(s._h, _pd(y), _pd(x), None, None, 1) == 0
    _check_forecast(y, sp, s.getDraws(), x, 7, 1, y_tol)
    s.close()
