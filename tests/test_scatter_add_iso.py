"""The sum of a scattering row's isotropic and anisotropic parts (radrhd_solver_b200/csrc/add_iso.h, compiled here
for the host): one rounding to float of the sum, whichever part is the larger and whatever their signs.  Bar: half
an ulp of the result and the terms of 2^-48 iso that two floats leave out (their split and the sum of the small
terms: 2^-47)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "radrhd_solver_b200", "csrc")
CODE = """#include "add_iso.h"
extern "C" void run(long n, const float *v, const double *iso, float *out) {
  for (long i = 0; i < n; i++) {
    const float hi = (float)iso[i], lo = fabsf(hi) < INFINITY ? (float)(iso[i] - (double)hi) : 0.f;
    out[i] = add_iso(v[i], hi, lo);
  }
}
"""


@pytest.fixture(scope="module")
def add(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("add_iso")
    (d / "a.cpp").write_text(CODE)
    subprocess.run([cxx, "-O2", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "a.so"), str(d / "a.cpp")], check=True)
    lib = C.CDLL(str(d / "a.so"))

    def run(v, iso):
        out = np.zeros_like(v)
        lib.run(C.c_long(v.size), *(C.c_void_p(a.ctypes.data) for a in (v, iso, out)))
        return out
    return run


@pytest.mark.parametrize("scale", [0.0, -0.3, 0.3, -2.0, 2.0, -7.0, 7.0, 20.0])
def test_one_rounding(add, scale):
    """scale: decades of the anisotropic part over the isotropic one."""
    rng = np.random.default_rng(7)
    n = 200_000
    iso = rng.uniform(1, 2, n) * 2.0 ** rng.integers(-30, 30, n) * rng.choice([-1, 1], n)
    v = (iso * rng.uniform(0.5, 2, n) * 10 ** scale * rng.choice([-1, 1], n)).astype(np.float32)
    got = add(v, iso)
    exact = v.astype(np.longdouble) + iso.astype(np.longdouble)
    bar = 0.5 * np.spacing(np.abs(got)).astype(np.longdouble) + 2.0 ** -47 * np.abs(iso)
    assert np.all(np.abs(got.astype(np.longdouble) - exact) <= bar)


def test_not_finite(add):
    v = np.array([np.inf, -np.inf, np.nan, 3e38, 1.0, 1.0, 0.0], np.float32)
    iso = np.array([1.0, 1.0, 1.0, 3e38, 1e300, -1e300, 0.0])
    assert np.array_equal(add(v, iso), np.array([np.inf, -np.inf, np.nan, np.inf, np.inf, -np.inf, 0.0], np.float32),
                          equal_nan=True)
