"""log|det| of FP64 draws by the deep elimination, against the oracle, at the edges of
its plan: dense parts of one node, of less than and more than a panel (16) or a warp
(32), of each block size, and the largest; and draws that it hands to the pivoting redo.

Tolerance: both are backward stable FP64 eliminations of matrices with condition
numbers below 100 and multipliers below 8; log|det| then has an error of a few
m * 2^-53, 1e-13 at m = 400; 1e-11 leaves two orders for growth.
"""
import numpy as np
import pytest

import oracle
from gpusgdlm_gb300 import SGDLM

pytestmark = pytest.mark.gpu


def _engine(m, kmax, seed, spread, n_ext=3):
    import bench

    wl = bench.make_workload(m=m, kmax=kmax, n_ext=n_ext, T=2, seed=seed)
    P = wl["P"]
    s = SGDLM(1, strict=True, precision="fp64")
    s.setSimultaneousParents(wl["p"], np.where(wl["sp"] >= m * m, np.nan, wl["sp"]).astype(float))
    s.setDiscountFactors(np.full(m, 0.97), np.full((P, P, m), 0.98))
    rng = np.random.default_rng(seed)
    a = rng.uniform(-spread, spread, size=(P, m))
    s.setPosteriorParameters(a, np.repeat((1e-6 * np.eye(P))[:, :, None], m, axis=2),
                             np.full(m, 50.0), np.full(m, 1.0))
    s.setRngState(seed, 0)
    return s, wl


@pytest.mark.parametrize("m,kmax,n", [
    (33, 1, 100), (40, 5, 3), (45, 17, 700), (64, 17, 300), (90, 12, 500), (130, 17, 200),
    (150, 30, 200), (230, 17, 160), (300, 17, 160), (400, 17, 200), (500, 6, 160)])
def test_log_dets_match_oracle(built_lib, m, kmax, n):
    s, wl = _engine(m, kmax, 7 + m, min(0.3, 0.8 / kmax))
    s.computeVBPosterior(n, n)
    assert s.getStats()["draws_pivoted"] == 0
    d = s.getDraws()
    k = min(n, 24)
    pick = np.r_[0:k // 2, n - (k - k // 2):n]
    ld = oracle.logdet(wl["sp"], np.asfortranarray(d["thetas"][:, :, pick].transpose(0, 2, 1)))
    np.testing.assert_allclose(d["log_dets"][pick], ld, rtol=0, atol=1e-11)
    s.close()


def test_draws_that_need_pivoting_are_redone(built_lib):
    """Coefficients up to 3: multipliers above the limit in most draws; the redo's
    partial pivoting loses a few more digits on these matrices."""
    m, n = 100, 64
    s, wl = _engine(m, 10, 5, 3.0)
    s.computeVBPosterior(n, n)
    assert s.getStats()["draws_pivoted"] > 0
    d = s.getDraws()
    ld = oracle.logdet(wl["sp"], np.asfortranarray(d["thetas"].transpose(0, 2, 1)))
    np.testing.assert_allclose(d["log_dets"], ld, rtol=0, atol=1e-8)
    s.close()
