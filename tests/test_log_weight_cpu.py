"""The log of a component's weight (tgmm_math.cuh, compiled for the host) against the separate
logarithms: an alpha that is negative, zero, not a number, tiny or huge, and determinants at the
ends of the range, where a product of them is not a normal number."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..")


@pytest.fixture(scope="module")
def log_weight(tmp_path_factory):
    d = tmp_path_factory.mktemp("weight")
    (d / "h.cpp").write_text('#include "tgmm_math.cuh"\n'
                             'extern "C" double f(double p, double a) { return tgmm::log_weight(p, a); }\n')
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "tgmm_b200", "csrc"),
                    str(d / "h.cpp"), "-o", str(d / "h.so")], check=True)
    f = C.CDLL(str(d / "h.so")).f
    f.restype, f.argtypes = C.c_double, [C.c_double, C.c_double]
    return f


@pytest.mark.parametrize("alpha", [-1e9, -3.0, -1e-200, 0.0, 1e-320, 1e-250, 1e-150, 1e-99, 1e-5, 1.0, 400.0, 1e9, 1e140,
                                   1e200, math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("p", [-1e-3, 0.0, 1e-320, 1e-300, 1e-200, 1e-12, 1.0, 1e7, 1e250, 1e305, math.inf, math.nan])
def test_log_weight_is_the_sum_of_its_logarithms(log_weight, p, alpha):
    with np.errstate(all="ignore"):
        parts = 0.5 * np.log(np.float64(p)), -1.5 * np.log(2 * np.pi), np.log(np.float64(alpha))
        want = sum(parts)
    got = log_weight(p, alpha)
    if not math.isfinite(want):
        assert got == want or (math.isnan(got) and math.isnan(want))
    else:
        # a few roundings of the largest term each
        assert abs(got - want) <= 4 * np.finfo(np.float64).eps * max(1.0, *map(abs, parts))
