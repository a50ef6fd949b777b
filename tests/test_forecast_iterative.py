"""The iterative forecast solves against the factorising path (which the other tests
compare with the oracle), at the edges of their launch rule: one draw per block, two
draws per block, a last block with a single draw, m at and beside multiples of 32,
more rows than the two-draw form takes, and values far outside FP32's range.

Tolerance of the FP64 form: both solve the same FP64 system with a backward error of
a few 2^-53 (growth below 8, condition numbers below 100 for these draws), so they
agree to 100 * 2^-53 * a few = 1e-13 of the draw's largest value; 1e-12 leaves a
factor of ten.
"""
import numpy as np
import pytest

import oracle
from gpusgdlm_gb300 import SGDLM

pytestmark = pytest.mark.gpu


def _engine(m, kmax, precision, seed=3, levels=4):
    import bench

    wl = bench.make_workload(m=m, kmax=kmax, T=4, seed=seed)
    P = wl["P"]
    s = SGDLM(1, strict=True, precision=precision)
    s.setSimultaneousParents(wl["p"], np.where(wl["sp"] >= m * m, np.nan, wl["sp"]).astype(float))
    s.setWarpLu(False)  # m <= 32 takes the warp path by default
    s.setDiscountFactors(np.full(m, 0.97), np.full((P, P, m), 0.98))
    rng = np.random.default_rng(seed)
    s.setPriorParameters(rng.uniform(-0.05, 0.05, size=(P, m)),
                         np.repeat((1e-4 * np.eye(P))[:, :, None], m, axis=2),
                         np.full(m, 20.0), np.full(m, 1.0))
    return s, wl


def _forecast(s, wl, n, x, iterative):
    s.setForecastSolver(iterative)
    s.setRngState(11, 0)
    return s.computeForecast(n, n, x)


@pytest.mark.parametrize("m,kmax,n,scale", [
    (3, 2, 5, 1.0), (32, 4, 1, 1.0), (33, 4, 4001, 1.0), (100, 10, 3000, 1e-250), (100, 10, 3000, 1e250),
    (129, 17, 2501, 1.0), (400, 17, 601, 1.0), (540, 5, 700, 1.0)])
def test_fp64_matches_factored(built_lib, m, kmax, n, scale):
    s, wl = _engine(m, kmax, "fp64")
    x = scale * wl["F_of"](2, False)
    y = _forecast(s, wl, n, x, True)
    assert s.getStats()["forecast_draws_factored"] == 0
    ref = _forecast(s, wl, n, x, False)
    assert s.getStats()["forecast_draws_factored"] == n
    err = np.abs(y - ref).max(axis=0) / np.abs(ref).max(axis=0)
    assert err.max() <= 1e-12
    s.close()


def test_fp64_log_dets_after_forecast(built_lib):
    """The draws' log|det| are not needed by the solve; getDraws still has them."""
    s, wl = _engine(70, 6, "fp64")
    n = 500
    _forecast(s, wl, n, wl["F_of"](2, False), True)
    d = s.getDraws()
    ld = oracle.logdet(wl["sp"], np.asfortranarray(d["thetas"].transpose(0, 2, 1)))
    np.testing.assert_allclose(d["log_dets"], ld, rtol=0, atol=1e-12)
    s.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("m", [33, 250, 520])
def test_draws_do_not_depend_on_their_block(built_lib, precision, m):
    """The same draw solved in a block of its own (few draws) and beside another one
    (many draws) gives the same bits."""
    s, wl = _engine(m, 6, precision)
    x = wl["F_of"](2, False)
    many = _forecast(s, wl, 4000, x, True)
    few = _forecast(s, wl, 3, x, True)
    np.testing.assert_array_equal(few, many[:, :3])
    s.close()


@pytest.mark.parametrize("m,kmax,mean", [(31, 4, 0.05), (447, 17, 0.05), (448, 20, 0.05), (449, 17, 0.05),
                                         (448, 17, 1e-40), (200, 8, 0.0)])
def test_fp32_two_blocks_per_sm(built_lib, m, kmax, mean):
    """FP32 draws at and beside the largest system of the form with two blocks on an SM,
    with Gamma entries below the normal FP32 numbers and at zero: both paths correct an FP32
    solve (relative error 2^-20 at most) by a solve of its FP64 residual, so they are within
    about 2^-30 of the solution; 1e-8 leaves a factor of five for each."""
    s, wl = _engine(m, kmax, "mixed")
    P = wl["P"]
    rng = np.random.default_rng(m)
    s.setPriorParameters(rng.uniform(-mean, mean, size=(P, m)),
                         np.repeat(((1e-4 if mean > 1e-9 else 1e-90) * np.eye(P))[:, :, None], m, axis=2),
                         np.full(m, 20.0), np.full(m, 1.0))
    x = wl["F_of"](2, False)
    y = _forecast(s, wl, 5001, x, True)
    assert s.getStats()["forecast_draws_factored"] == 0
    ref = _forecast(s, wl, 5001, x, False)
    err = np.abs(y - ref).max(axis=0) / np.abs(ref).max(axis=0)
    assert err.max() <= 1e-8
    s.close()


@pytest.mark.parametrize("m,kmax,n,scale,own", [
    (40, 4, 300, 1e-6, 0.1), (100, 6, 2000, 1e-8, 0.12), (400, 8, 320, 1e-5, 0.1), (540, 5, 100, 1e-7, 0.1)])
def test_fp64_series_of_different_scales(built_lib, m, kmax, n, scale, own):
    """Half of the series are `scale` as large as the others, depend on each other only and
    converge more slowly: their forecasts are as exact as the large ones'.  Error of each
    value against the size of the terms it is the sum of, |nu_r| + sum |gamma_rq y_q|; the
    bound is the file's 1e-12."""
    half = m // 2
    rng = np.random.default_rng(m)
    P = kmax + 1
    sp = np.full((P, m), 2147483648, dtype=np.uint32, order="F")
    a = np.zeros((P, m))
    for j in range(m):
        block = np.arange(half) if j < half else np.arange(half, m)
        sp[1:, j] = j + m * rng.choice(block[block != j], size=kmax, replace=False)
        a[1:, j] = rng.uniform(-0.01, 0.01, kmax) if j < half else own * rng.choice([0.7, 1.0], kmax)
    s = SGDLM(1, strict=True, precision="fp64")
    s.setSimultaneousParents(np.full(m, P), np.where(sp >= m * m, np.nan, sp).astype(float))
    s.setDiscountFactors(np.full(m, 0.97), np.full((P, P, m), 0.98))
    s.setPriorParameters(a, np.repeat((1e-8 * np.eye(P))[:, :, None], m, axis=2), np.full(m, 20.0),
                         np.where(np.arange(m) < half, 1.0, scale**2))
    x = np.zeros((P, m))
    wl = dict(P=P)
    y = _forecast(s, wl, n, x, True)
    assert s.getStats()["forecast_draws_factored"] == 0
    th = s.getDraws()["thetas"]
    ref = _forecast(s, wl, n, x, False)
    G = np.zeros((n, m, m))
    for j in range(m):
        G[:, j, sp[1:, j] // m] = th[1:, j, :].T
    nu = np.abs(ref.T - np.einsum("irq,qi->ir", G, ref))
    size = nu + np.einsum("irq,qi->ir", np.abs(G), np.abs(ref))
    assert (np.abs(y - ref).T / size).max() <= 1e-12
    s.close()


def test_fp64_rows_that_cancel(built_lib):
    """Rows whose terms nearly cancel in a neighbour do not send a draw to the LU: the
    bench's kind of system, 40 000 draws (one in 10 000 has such a row), against the
    factored solves."""
    m, n = 60, 40000
    s, wl = _engine(m, 17, "fp64")
    P = wl["P"]
    rng = np.random.default_rng(8)
    s.setPriorParameters(rng.normal(0, 0.06, size=(P, m)), np.repeat((1e-4 * np.eye(P))[:, :, None], m, axis=2),
                         np.full(m, 20.0), np.full(m, 1.0))
    x = wl["F_of"](2, False)
    y = _forecast(s, wl, n, x, True)
    assert s.getStats()["forecast_draws_factored"] == 0
    ref = _forecast(s, wl, n, x, False)
    err = np.abs(y - ref).max(axis=0) / np.abs(ref).max(axis=0)
    assert err.max() <= 1e-12
    s.close()


@pytest.mark.parametrize("m,rows", [(447, 8), (448, 8), (449, 8), (384, 12), (385, 12), (385, 18), (385, 20),
                                    (510, 24), (512, 30), (513, 30)])
def test_two_draws_per_block(built_lib, m, rows):
    """FP32 draws at and beside the sizes where a block takes two: the same bits as a few
    draws one by one, up to an odd last one."""
    s, wl = _engine(m, rows, "mixed", seed=m)
    x = wl["F_of"](2, False)
    many = _forecast(s, wl, 2501, x, True)
    assert s.getStats()["forecast_draws_factored"] == 0
    few = _forecast(s, wl, 5, x, True)
    np.testing.assert_array_equal(few, many[:, :5])
    s.setForecastSolver(True)
    s.setRngState(11, 0)
    odd = s.computeForecast(2500, 2500, x)
    np.testing.assert_array_equal(odd, many[:, :2500])
    s.close()
