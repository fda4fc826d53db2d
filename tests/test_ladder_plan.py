"""Task lists of the ladder kernels, checked on the host: tests/ladder_plan_check.cu includes the plan builders
and walks every list as the kernels do, for Pauli sums from none to a few thousand words."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path_factory.mktemp("ladder") / "ladder_plan_check.so"
    res = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC",
                          "-shared", str(HERE / "ladder_plan_check.cu"), "-o", str(out)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    lib = ctypes.CDLL(str(out))
    lib.check_ladder_plan.restype = ctypes.c_longlong

    def run(codes, mirror=0, real=1, layers=4):
        codes = np.ascontiguousarray(codes, dtype=np.uint8)
        T, n = codes.shape
        coeffs = np.ones(max(T, 1))
        msg = ctypes.create_string_buffer(200)
        steps = lib.check_ladder_plan(n, T, codes.ctypes.data_as(ctypes.c_void_p), coeffs.ctypes.data_as(ctypes.c_void_p),
                                      mirror, real, layers, msg, 200)
        return steps, msg.value.decode()
    run.lib = lib
    return run


def _words(rng, n, count, weight):
    codes = np.zeros((count, n), dtype=np.uint8)
    for row in codes:
        at = rng.permutation(n)[:rng.integers(1, min(weight, n) + 1)]
        row[at] = rng.integers(1, 4, at.size)
    return codes


@pytest.mark.parametrize("real", [1, 0])
@pytest.mark.parametrize("mirror", [0, 1])
def test_lists_stay_inside_their_arrays(check, mirror, real):
    rng = np.random.default_rng(3)
    sums = [np.zeros((0, 5)), np.zeros((2, 4)), np.eye(6), 2 * np.eye(3), np.full((1, 7), 3)]
    sums += [_words(rng, n, count, weight) for n in (2, 3, 9, 40, 96) for count in (1, 17, 300) for weight in (1, 4, n)]
    sums.append(_words(rng, 64, 4000, 6))
    for codes in sums:
        for layers in (1, 4):
            steps, fault = check(codes, mirror, real, layers)
            assert steps >= 0, (codes.shape, layers, fault)


def test_passes_stay_inside_their_budget(check):
    size = ctypes.c_ulonglong
    for state in (1, 1000, 3 << 30):
        for states in (0, 1, 2, 7, 8, 9, 15, 16, 100):
            for B in (1, 5, 8, 40):
                n = check.lib.check_ladder_pass(B, size(state), size(states * state + state // 2))
                assert 1 <= n <= B and (n <= max(states, 1))
                assert n == B or n == (states & ~7 if states >= 8 else max(states, 1))
