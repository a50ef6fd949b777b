"""Errors of the FP64 logarithm, sine and cosine by table (no GPU: the header's operations,
which the device rounds alike, against long double).

Bounds, as the header derives them: logarithm 1/2 ulp for the last addition, 2^-59 of the
polynomial relative to the result (2^-6 ulp), and less than 2^-10 ulp of the parts below:
0.517 ulp; sine and cosine 2^-54 for the table's value, 2^-54 for the last addition and
2^-60 for the products: 1.12e-16.
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
LOG_ULP, TRIG_ABS = 0.517, 1.12e-16


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("trig") / "libtrig_log.so"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                        str(ROOT / "tests" / "trig_log_check.cpp"), "-o", str(out)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(out))


def _run(f, a, dtype):
    a = np.ascontiguousarray(a, dtype=dtype)
    out = np.zeros(len(a))
    f(C.c_long(len(a)), a.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
    return out


def _uniforms():
    """Both ends, the values about every interval's edges in every binade, and random ones."""
    rng = np.random.default_rng(1)
    a = [np.arange(20000), 2**32 - 1 - np.arange(20000), rng.integers(0, 2**32, 300000)]
    for e in range(9, 33):  # v = 2 a + 1 in [2^e, 2^(e + 1))
        edge = (2**e + np.arange(257) * 2**e // 256) // 2
        a += [edge + d for d in (-1, 0, 1)]
    a = np.concatenate(a)
    return a[(a >= 0) & (a < 2**32)]


def test_log_of_uniforms(lib):
    assert _run(lib.check_log_uniform, _uniforms(), np.uint32).max() <= LOG_ULP


@pytest.mark.parametrize("k", [-1022, -700, -32, -2, -1, 0, 1, 5, 1023])
def test_log(lib, k):
    rng = np.random.default_rng(k & 0xFFFF)
    edge = 1 + np.arange(256) / 256
    m = np.concatenate([edge, np.nextafter(edge, 2), np.nextafter(edge[1:], 0), rng.uniform(1, 2, 100000),
                        1 + 2.0**-52 * np.arange(1, 200), 2 - 2.0**-52 * np.arange(1, 200),
                        1 + 2.0**-rng.uniform(8, 52, 5000), 2 - 2.0**-rng.uniform(7, 51, 5000)])
    x = np.ldexp(m[m < 2], k)
    assert _run(lib.check_log, x, np.float64).max() <= LOG_ULP


def test_log_of_special_values(lib):
    x = np.array([0.0, -0.0, 5e-324, 2.0**-1030, 2.2250738585072014e-308, 1.0, 1.7976931348623157e308,
                  np.inf, -1.0, -np.inf, np.nan])
    with np.errstate(all="ignore"):
        want = np.log(x)
    np.testing.assert_allclose(_run(lib.values_log, x, np.float64), want, rtol=2.3e-16, atol=0)


def test_sin_and_cos(lib):
    rng = np.random.default_rng(2)
    # every angle of the table, and the ends and the middles of its neighbourhood (2^22
    # units of 2 pi 2^-33 to either side)
    at = (np.arange(1025) * 2**23)[:, None] + np.array([-2**22, -2**22 + 1, -1, 1, 2**22 - 1, 2**22])
    b = np.concatenate([at.ravel() // 2, rng.integers(0, 2**32, 300000), np.arange(1000),
                        2**32 - 1 - np.arange(1000)])
    b = b[(b >= 0) & (b < 2**32)]
    assert _run(lib.check_sincos, b, np.uint32).max() <= TRIG_ABS
