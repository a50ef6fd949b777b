"""Host model of the block-wide maxima with one barrier each (no GPU): warps in any
order never lose a maximum or read a stale one under the rules of
gpusgdlm_gb300/csrc/max_sets.hpp, where two sets used in turn do."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    out = tmp_path_factory.mktemp("max_sets") / "libmax_sets.so"
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC",
                        str(ROOT / "tests" / "max_sets_check.cpp"), "-o", str(out)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(str(out))
    L.max_sets_run.restype = C.c_long
    L.max_sets_run.argtypes = [C.c_int, C.c_int, C.c_int, C.c_uint64]
    return L


@pytest.mark.parametrize("warps", [1, 2, 3, 14, 32])
def test_no_maximum_is_lost(model, warps):
    assert sum(model.max_sets_run(warps, 40, 0, seed) for seed in range(1, 200)) == 0


def test_two_sets_lose_maxima(model):
    assert sum(model.max_sets_run(4, 40, 1, seed) for seed in range(1, 200)) > 0
