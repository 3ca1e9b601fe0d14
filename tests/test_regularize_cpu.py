"""The device form of the precision regularisation (reciprocals, ratios as products; tgmm_math.cuh
compiled for the host with the device's branches) against its plain form, which divides: over
anisotropic and nearly spherical matrices, with nu of either sign."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..")
HARNESS = r"""
#include <math.h>
static inline double rsqrt(double x) { return 1.0 / sqrt(x); }
#include "tgmm_math.cuh"
extern "C" void run(double* W, double nu, const float* scale, int w4dof, const double* lim) {
  tgmm::RegConst rc;
  double inv[6];
  for (int i = 0, e = 0; i < 3; i++)
    for (int j = i; j < 3; j++) inv[e++] = 1.0 / (double)(scale[i] * scale[j]);
  for (int d = 0; d < 3; d++) rc.scale[d] = scale[d];
  rc.w4dof = w4dof, rc.lambda_min = lim[0], rc.lambda_max = lim[1], rc.max_exc = lim[2], rc.inv_s2 = inv;
  tgmm::regularize_W(W, nu, rc);
}
"""


@pytest.fixture(scope="module")
def forms(tmp_path_factory):
    d = tmp_path_factory.mktemp("reg")
    (d / "h.cpp").write_text(HARNESS)
    out = []
    for name, flags in (("plain", []), ("device", ["-D__CUDA_ARCH__=1000"])):
        subprocess.run(["g++", "-std=gnu++17", "-O2", "-shared", "-fPIC", *flags,
                        "-I" + os.path.join(ROOT, "tgmm_b200", "csrc"), str(d / "h.cpp"), "-o", str(d / (name + ".so"))],
                       check=True)
        f = C.CDLL(str(d / (name + ".so"))).run

        def call(W, nu, scale, w4, lim, f=f):
            w = np.array(W, np.float64)
            f(w.ctypes.data_as(C.c_void_p), C.c_double(nu), np.array(scale, np.float32).ctypes.data_as(C.c_void_p),
              C.c_int(w4), np.array(lim, np.float64).ctypes.data_as(C.c_void_p))
            return w
        out.append(call)
    return out


@pytest.mark.parametrize("w4", [0, 1])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("max_exc", [0.5, 1.0, 3.0, 9.0])
def test_device_form_gives_the_plain_forms_matrix(forms, w4, sign, max_exc):
    plain, device = forms
    rng = np.random.default_rng(int(10 * max_exc) + w4)
    for _ in range(300):
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        lam = np.exp(rng.uniform(np.log(0.005), np.log(0.5), 3))
        nu = sign * np.exp(rng.uniform(0, 8))
        W = (q * (lam / nu)) @ q.T
        args = (W[np.triu_indices(3)], nu, (1.0, 1.0, 5.0), w4, (0.02, 0.2222, max_exc))
        a, b = plain(*args), device(*args)
        # the closed-form eigenvectors lose about half the digits where two eigenvalues meet
        assert np.max(np.abs(a - b)) <= 1e-7 * np.max(np.abs(a)), (a, b)
