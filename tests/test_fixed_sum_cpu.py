"""The log-likelihood's order-free sums (tgmm_math.cuh, compiled for the host): a frame of many more
parts than one 64-bit word of 2^-40 fractions holds keeps its total, whatever the lanes' shares,
and the total is the exact one of the parts' fixed-point values."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..")
HARNESS = r"""
#include "tgmm_math.cuh"
using namespace tgmm;
// `warps` warps of 32 lanes, each lane with `parts` parts v and `dropped` of them subtracted again,
// summed as the voxel pass does; the exact total of the kept ones in units of 2^-40.
extern "C" void run(int warps, long long parts, long long dropped, double v, int carry, double* got, long long* exact_hi,
                    unsigned long long* exact_lo) {
  long long fi = 0, i1 = 0;
  unsigned long long ff = 0, f1 = 0;
  fixed_acc(i1, f1, v);
  for (int w = 0; w < warps; w++) {
    long long wi = 0;
    unsigned long long wf = 0;
    for (int l = 0; l < 32; l++) {
      long long ai = 0, di = 0;
      unsigned long long ar = 0, dr = 0;
      for (long long p = 0; p < parts; p++) {
        fixed_acc(ai, ar, v);
        if (p < dropped) di -= i1, dr -= f1;
      }
      if (carry && parts > 2048) fixed_carry(ai, ar), fixed_carry(di, dr);  // as after a large supervoxel
      ai += di, ar += dr;
      wi += ai, wf += ar;
    }
    if (carry) fixed_carry(wi, wf);
    fi += wi, ff += wf;
  }
  if (carry) fixed_carry(fi, ff);
  *got = (double)fi + (double)ff / kFracScale;
  const __int128 n = (__int128)warps * 32 * (parts - dropped), x = n * (((__int128)i1 << 40) + (__int128)f1);
  *exact_hi = (long long)(x >> 64);
  *exact_lo = (unsigned long long)x;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "tgmm_b200", "csrc"),
                    str(d / "h.cpp"), "-o", str(d / "h.so")], check=True)
    f = C.CDLL(str(d / "h.so")).run

    def call(warps, parts, dropped, v, carry=1):
        got, hi, lo = C.c_double(), C.c_int64(), C.c_uint64()
        f(C.c_int(warps), C.c_int64(parts), C.c_int64(dropped), C.c_double(v), C.c_int(carry), C.byref(got),
          C.byref(hi), C.byref(lo))
        return got.value, (hi.value << 64) + lo.value
    return call


@pytest.mark.parametrize("v", [0.9999999999, -0.25, -4321.0000001, 17.5])
@pytest.mark.parametrize("warps,parts,dropped", [(1, 1, 0), (3, 40, 7), (2368, 300, 0), (2368, 300, 299), (4, 200000, 3)])
def test_total_beyond_one_word_of_fractions(run, warps, parts, dropped, v):
    got, exact = run(warps, parts, dropped, v)
    assert got == exact / 2 ** 40  # one rounding of the exact total


def test_without_the_carry_it_would_wrap(run):
    """22.7 M parts near one: more than 2^24."""
    got, exact = run(2368, 300, 0, 0.9999999999, carry=0)
    assert exact / 2 ** 40 - got == pytest.approx(2.0 ** 24)
