"""Integer sums and quotients of the Krylov scalars (gsls_fixsum.cuh) against
exact arithmetic, on the host: the functions are the ones the kernels use.

Bounds, from the header: an addend is cut at 2^-68 of the largest one, a total
is rounded to nearest once (half a unit in the last place), a quotient is
within 0.51 units in the last place.
"""
import ctypes as C
import math
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]

# the sum as grid_red_total takes it: `per` addends a lane and turn, one
# partial per addend (blocks of one value)
SHIM = r"""
#include <string.h>
#include "gsls_fixsum.cuh"
using namespace gsls;
static unsigned long long bits(double v) { unsigned long long u; memcpy(&u, &v, 8); return u; }
extern "C" double sum(const double *v, int n, int per) {
  long long T = 0, H[32] = {0};
  unsigned L = 0, Lo[32] = {0};
  int E = 1;
  for (int k0 = 0; k0 < n; k0 += 32 * per) {
    int e = E;
    for (int k = k0; k < n && k < k0 + 32 * per; k++) {
      const int x = fix_exp(bits(v[k]));
      if (x > e) e = x;
    }
    for (int l = 0; l < 32; l++) {
      if (k0 > 0 && e > E) {
        int lo = (int)Lo[l];
        fix_down(H[l], lo, e - E);
        Lo[l] = (unsigned)lo;
      }
      for (int k = 0; k < per; k++) {
        const int i = k0 + l + 32 * k;
        if (i >= n) continue;
        int S[3], lo, own = fix_exp(bits(v[i]));
        long long hi;
        if (own < 1) own = 1;
        fix_limbs(bits(v[i]), own, S);
        fix_align(own, S, e, hi, lo);
        H[l] += hi;
        Lo[l] += (unsigned)lo;
      }
      H[l] += Lo[l] >> 23;
      Lo[l] &= kFixMask;
    }
    E = e;
  }
  for (int l = 0; l < 32; l++) { T += H[l]; L += Lo[l]; }
  return fix_double(T, L, E);
}
extern "C" double quot(double a, double b) { return fix_div(a, b); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    inc = next((p for p in ("/usr/local/cuda/include", "/usr/local/cuda/targets/x86_64-linux/include")
                if Path(p, "cuda_runtime.h").exists()), None)
    if inc is None or shutil.which("g++") is None:
        pytest.skip("no CUDA headers or host compiler")
    d = tmp_path_factory.mktemp("fixsum")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{inc}",
                    f"-I{ROOT / 'svfsi_gb300' / 'csrc'}", str(d / "shim.cpp"), "-o",
                    str(d / "shim.so")], check=True)
    L = C.CDLL(str(d / "shim.so"))
    L.sum.restype = L.quot.restype = C.c_double
    L.sum.argtypes = [C.POINTER(C.c_double), C.c_int, C.c_int]
    L.quot.argtypes = [C.c_double, C.c_double]
    return L


def _check_sum(lib, v, per=5):
    v = np.ascontiguousarray(v, float)
    got = lib.sum(v.ctypes.data_as(C.POINTER(C.c_double)), v.size, per)
    exact = sum((Fraction(float(x)) for x in v), Fraction(0))
    cut = Fraction(float(np.abs(v).max())) * v.size / 2 ** 68
    half = Fraction(math.ulp(float(exact))) / 2
    assert abs(Fraction(got) - exact) <= half + 2 * cut, (got, float(exact))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 152, 160, 161, 256])
@pytest.mark.parametrize("spread", [0, 5, 22, 23, 24, 46, 80])
def test_sums(lib, n, spread):
    rng = np.random.default_rng(n + spread)
    for scale in (1.0, 1e-200, 1e200):
        v = rng.standard_normal(n) * 2.0 ** rng.integers(-spread, 1, n) * scale
        _check_sum(lib, v)
        _check_sum(lib, np.concatenate([v, -v[: n // 2]])[:256])


@pytest.mark.parametrize("shift", [1, 10, 22, 23, 30, 40, 46, 60])
def test_earlier_turn_keeps_its_digits(lib, shift):
    """The largest values come in the second turn and cancel there."""
    rng = np.random.default_rng(shift)
    small = rng.standard_normal(160) * 2.0 ** -shift
    big = rng.standard_normal(48)
    _check_sum(lib, np.concatenate([small, big, -big]))


def test_quotients(lib):
    rng = np.random.default_rng(3)
    a = rng.uniform(1, 2, 4000) * 2.0 ** rng.integers(-300, 300, 4000) * rng.choice([-1, 1], 4000)
    b = rng.uniform(1, 2, 4000) * 2.0 ** rng.integers(-300, 300, 4000) * rng.choice([-1, 1], 4000)
    edge = [1.0, 1.5, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52, 3.0, -1.0]
    pairs = list(zip(a, b)) + [(x, y) for x in edge for y in edge] + [(x, x) for x in a[:200]]
    for x, y in pairs:
        q = Fraction(float(x)) / Fraction(float(y))
        assert abs(Fraction(lib.quot(x, y)) - q) <= Fraction(51, 100) * Fraction(math.ulp(float(q)))


def test_quotients_of_special_values(lib):
    inf, nan, sub = math.inf, math.nan, 5e-324
    vals = [0.0, -0.0, 1.0, -3.0, inf, -inf, nan, sub, 1e-308, 1e308, -1e308]
    with np.errstate(all="ignore"):
        for x in vals:
            for y in vals:
                want = float(np.float64(x) / np.float64(y))
                got = lib.quot(x, y)
                assert (math.isnan(got) and math.isnan(want)) or got == want, (x, y, got, want)
