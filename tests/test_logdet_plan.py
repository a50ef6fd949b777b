"""Host-side check (no GPU) of the plan for log|det| of FP64 draws and of the levels as a
stream of words per thread, evaluated in FP64 against a dense log|det|; and of both that
threads between two barriers touch no slot that another one writes.

Tolerance: FP64 eliminations without pivoting of matrices with coefficients N(0, 0.1^2)
(as test_elimination_plan.py: 1e-10).
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
NONE, MAX_SLOTS = 2147483648, 28928


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("plan") / "liblogdet_plan.so"
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-x", "c++",
                        str(ROOT / "tests" / "logdet_plan_check.cpp"), "-I", "/usr/local/cuda/include",
                        "-o", str(out)], capture_output=True, text=True)
    if r.returncode != 0 and "cuda_runtime.h" in r.stderr:
        pytest.skip("no CUDA headers")
    assert r.returncode == 0, r.stderr
    L = C.CDLL(str(out))
    L.logdet_plan_check.restype = L.level_stream_check.restype = C.c_double
    return L


def _sp(m, P):
    return np.full((P, m), NONE, dtype=np.uint32, order="F")


def _random(m, kmax, seed, P=None):
    rng = np.random.default_rng(seed)
    sp = _sp(m, P or kmax + 3)
    for j in range(m):
        q = rng.choice(np.delete(np.arange(m), j), size=min(m - 1, rng.integers(0, kmax + 1)), replace=False)
        sp[:len(q), j] = j + m * q
    return sp


def _full_row(m, r):
    """Series r has every other one as a parent, the others one each."""
    sp = _sp(m, m)
    others = np.delete(np.arange(m), r)
    sp[:m - 1, r] = r + m * others
    for j in others:
        sp[0, j] = j + m * ((j + 1) % m)
    return sp


def _full_col(m, c):
    """Every other series has c as a parent, and its neighbour."""
    sp = _sp(m, 2)
    for j in range(m):
        q = [v for v in (c, (j + 1) % m) if v != j]
        sp[:len(set(q)), j] = [j + m * v for v in dict.fromkeys(q)]
    return sp


def _any_rows(m, count, seed):
    """Entries at any off-diagonal position, not in their series' row."""
    rng = np.random.default_rng(seed)
    pos = np.array([r + m * c for r in range(m) for c in range(m) if r != c])
    P = -(-count // m)
    sp = np.full(P * m, NONE, dtype=np.uint32)
    sp[:count] = rng.permutation(pos)[:count]
    return np.asfortranarray(sp.reshape(P, m))


CASES = {
    "m1": _sp(1, 1), "m2_none": _sp(2, 1), "m2": _random(2, 1, 1), "m3": _random(3, 2, 2),
    "none": _sp(50, 3), "chain": _random(60, 1, 3), "m40": _random(40, 6, 4), "m100": _random(100, 10, 5),
    "m250": _random(250, 17, 6), "m400": _random(400, 17, 7), "dense": _random(45, 44, 8, P=44),
    "row": _full_row(70, 5), "column": _full_col(90, 17), "other_rows": _any_rows(60, 250, 9)}


def _want(sp, theta):
    P, m = sp.shape
    A = np.eye(m)
    for j in range(m):
        for k in range(P):
            if sp[k, j] < m * m:
                A[sp[k, j] % m, sp[k, j] // m] = -theta[j * P + k]
    return np.linalg.slogdet(A)[1]


def _call(f, sp, theta, *args):
    P, m = sp.shape
    info = np.zeros(4, dtype=np.int32)
    v = f(C.c_int(m), C.c_int(P), sp.ctypes.data_as(C.c_void_p), theta.ctypes.data_as(C.c_void_p),
          *[C.c_int(a) for a in args], info.ctypes.data_as(C.c_void_p))
    return v, info


def _theta(sp):
    return np.random.default_rng(sp.size).normal(0, 0.1, sp.size)


@pytest.mark.parametrize("name", CASES)
def test_logdet_plan(lib, name):
    sp = CASES[name]
    theta = _theta(sp)
    got, (core, levels, slots, sound) = _call(lib.logdet_plan_check, sp, theta, MAX_SLOTS)
    assert core >= 1 and sound
    np.testing.assert_allclose(got, _want(sp, theta), rtol=1e-10, atol=1e-10)


def test_logdet_plan_under_a_slot_limit(lib):
    """Slots are handed on; with too few of them there is no plan."""
    sp = CASES["m250"]
    theta = _theta(sp)
    _, (_, _, slots, _) = _call(lib.logdet_plan_check, sp, theta, MAX_SLOTS)
    for limit, planned in ((slots, True), (slots - 1, False), (250, False)):
        got, (core, _, used, sound) = _call(lib.logdet_plan_check, sp, theta, int(limit))
        assert (core > 0) == planned
        if planned:
            assert sound and used <= limit
            np.testing.assert_allclose(got, _want(sp, theta), rtol=1e-10, atol=1e-10)


@pytest.mark.parametrize("lanes", [128, 256])
@pytest.mark.parametrize("levels", [0, 1, 4, 16])
@pytest.mark.parametrize("name", CASES)
def test_level_stream(lib, name, levels, lanes):
    sp = CASES[name]
    theta = _theta(sp)
    got, (core, nlev, _, sound) = _call(lib.level_stream_check, sp, theta, levels, lanes)
    assert core >= 1 and nlev <= levels and sound
    np.testing.assert_allclose(got, _want(sp, theta), rtol=1e-10, atol=1e-10)
