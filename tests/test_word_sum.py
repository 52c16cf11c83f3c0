"""The running sum of the resident lead field (csrc/word_sum.h) on the CPU, against exact sums."""
import ctypes
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("needs g++")
    out = str(tmp_path_factory.mktemp("word_sum") / "word_sum.so")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-shared", "-fPIC", "-I",
                        os.path.join(ROOT, "ekgsim_gb300", "csrc"), os.path.join(ROOT, "tests", "native", "word_sum.cpp"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(out)
    for f in (lib.word_sum, lib.word_sum_short, lib.word_sum_parts):
        f.restype = ctypes.c_float
        f.argtypes = [ctypes.c_void_p, ctypes.c_int]
    return lib


def cancelling(rng, n):
    """Terms of both signs over three decades in pairs that cancel, in any order, and one of 2^-36 of them."""
    half = (rng.standard_normal(n // 2) * 10.0 ** rng.uniform(-2, 1, size=n // 2)).astype(np.float32)
    rest = (2.0**-36 * rng.standard_normal(n - 2 * half.size)).astype(np.float32)
    return rng.permutation(np.concatenate([half, -half, rest])).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 3, 17, 65, 512])
def test_no_more_is_lost_than_in_64_bits(lib, n):
    """Within half a unit of the result's last place (2^-24, and again for the last two additions) and the words'
    n^3 2^-72 of the terms' sum of magnitudes, which is below the n 2^-53 of a sum in FP64."""
    rng = np.random.Generator(np.random.PCG64(n))
    for _ in range(400):
        w = cancelling(rng, n)
        want = math.fsum(w.astype(np.float64))
        size = math.fsum(np.abs(w.astype(np.float64)))
        got = lib.word_sum(w.ctypes.data, n)
        assert lib.word_sum_short(w.ctypes.data, n) == got
        assert abs(got - want) <= 2.0**-23 * abs(want) + n**3 * 2.0**-72 * size


@pytest.mark.parametrize("n", [513, 2001, 20001])
def test_parts_in_64_bits(lib, n):
    """More terms than the words take: within the FP64 sum's bound, n 2^-53 of the terms' sum of magnitudes."""
    rng = np.random.Generator(np.random.PCG64(n))
    for _ in range(60):
        w = cancelling(rng, n)
        want = math.fsum(w.astype(np.float64))
        size = math.fsum(np.abs(w.astype(np.float64)))
        got = lib.word_sum_parts(w.ctypes.data, n)
        assert abs(got - want) <= 2.0**-24 * abs(want) + n * 2.0**-53 * size


@pytest.mark.parametrize("w,want", [([1, math.inf, 2], math.inf), ([-math.inf, 3], -math.inf),
                                    ([math.inf, -math.inf], math.nan), ([1, math.nan], math.nan), ([-0.0], 0.0)])
def test_not_finite(lib, w, want):
    a = np.array(w, dtype=np.float32)
    for f in (lib.word_sum, lib.word_sum_short, lib.word_sum_parts):
        got = f(a.ctypes.data, a.size)
        assert (math.isnan(want) and math.isnan(got)) or got == want
