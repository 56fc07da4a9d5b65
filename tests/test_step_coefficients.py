"""Host code of the FP32 steps' interface (psv_tma.hpp), compiled on its own.

The resident step's FP32 stencil coefficients (SimDesc::set_steps): the difference of a linear field is the step h to 2^-27, the
rounding of three times the small coefficient (three halves of a unit in the
last place of h / 24, at most 2^-24 relative), and that of a cubic field
vanishes to 2^-20 (27/3 times the large coefficient's rounding, 9/8 2^-24)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from psvwave_gb300 import build

SOURCE = """
#include "psv_tma.hpp"
extern "C" void coefficients(double dt, double dx, double dz, float *out) {
  psv::tma::SimDesc d;
  d.set_steps(dt, dx, dz);
  for (int k = 0; k < 4; ++k) out[k] = d.coef[k];
}
extern "C" const char *wait_error(int flags) { return psv::tma::wait_error(flags); }
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    folder = tmp_path_factory.mktemp("coef")
    src, lib = str(folder / "coef.cpp"), str(folder / "coef.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", build.CSRC, "-I", include, src,
                    "-o", lib], check=True)
    return ctypes.CDLL(lib)


@pytest.fixture(scope="module")
def coefficients(library):
    fn = library.coefficients
    fn.argtypes = [ctypes.c_double] * 3 + [ctypes.c_void_p]

    def call(dt, dx, dz):
        out = np.zeros(4, np.float32)
        fn(dt, dx, dz, out.ctypes.data)
        return out.astype(np.float64)
    return call


def test_differences_of_linear_fields_keep_the_step(coefficients):
    rng = np.random.default_rng(0)
    cases = [(2e-4, 1.249, 1.249), (2.5e-4, 1.249, 1.3), (4e-4, 5.0, 5.0)]
    cases += [tuple(10.0 ** rng.uniform((-6, -1, -1), (-2, 2, 2))) for _ in range(2000)]
    for dt, dx, dz in cases:
        a = coefficients(dt, dx, dz)
        for a1, a2, h in ((a[0], a[1], dt / dx), (a[2], a[3], dt / dz)):
            assert abs(a1 - 3 * a2 - h) <= 2.0 ** -27 * h
            assert abs(a1 - 27 * a2) <= 2.0 ** -20 * h


def test_a_wait_that_ran_out_is_named_by_its_flag(library):
    library.wait_error.restype = ctypes.c_char_p
    named = {f: library.wait_error(f) for f in range(1, 8)}
    assert b"copies" in named[1] and b"tiles" in named[2]
    assert all(b"resident" in named[f] for f in (4, 5, 6, 7))
