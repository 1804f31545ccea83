"""The FP64 quotients that stand in for IEEE divisions, from the header that the kernels include.

div_by, WScale and recips are compiled for the host and compared with IEEE division bit for bit over
random operands and the constants and extremes the reconstruction meets (all equal: they can differ
only where the exact value lies within 1e-15 ulp of the middle of two doubles, which no random operand
does).  sdiv starts from the device's refined reciprocal, which a GPU test takes from the device."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from helpers import make_torus
from harm_harm_b200 import Harm

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include <math.h>
#define __fdividef(a, b) ((a) / (b))
#define __ldg(p) (*(p))
#include "harm_device.cuh"
extern "C" void quotients(long n, const double* a, const double* b, double* div, double* scale) {
  for (long i = 0; i < n; i++) {
    const hb::WScale<double> s(b[i]);
    div[i] = hb::div_by(a[i], b[i], 1.0 / b[i]);
    scale[i] = s(a[i]);
  }
}
extern "C" void reciprocals(long n, const double* a, const double* b, const double* c, double* two, double* three) {
  for (long i = 0; i < n; i++) {
    hb::recips(a[i], b[i], two[i], two[n + i]);
    hb::recips(a[i], b[i], c[i], three[i], three[n + i], three[2 * n + i]);
  }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "harm_harm_b200", "csrc"), "-I", "/usr/local/cuda/include", "-o", str(d / "q.so"), str(d / "q.cpp")],
                   check=True, capture_output=True)
    return C.CDLL(str(d / "q.so"))


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def test_quotients_are_ieee(lib):
    rng = np.random.default_rng(5)
    n = 400000
    b = 10.0 ** rng.uniform(-150, 150, n)
    b[: n // 2] = rng.uniform(1.0, 2.0, n // 2)
    third = 1.0 / 3.0
    b[:7] = [12.0, 1.6 - 1.3, 0.8 * third - 0.2 * third, 1.0 - 1.2 * third, 2.2250738585072014e-308, 1.0 + 2.0**-52, 2.0 - 2.0**-52]
    a = rng.uniform(-1.0, 1.0, n) * b * 10.0 ** rng.uniform(-9, 3, n)
    a[7:9] = 0.0
    div, scale = np.empty(n), np.empty(n)
    lib.quotients(C.c_long(n), _p(a), _p(b), _p(div), _p(scale))
    assert np.array_equal(div, a / b) and np.array_equal(scale, a / b)


def test_shared_reciprocals_are_ieee(lib):
    """Over the range of the WENO sums' operands: (beta + 1e-26)^2 of measures that sum to one, and
    weight sums, down to the smallest product that stays normal."""
    rng = np.random.default_rng(6)
    n = 400000
    x = [10.0 ** rng.uniform(-52, 1, n) for _ in range(3)]
    for v in x:
        v[: n // 2] = rng.uniform(0.02, 2.0, n // 2)
    two, three = np.empty((2, n)), np.empty((3, n))
    lib.reciprocals(C.c_long(n), *(_p(v) for v in x), _p(two), _p(three))
    for k in range(3):
        assert np.array_equal(three[k], 1.0 / x[k])
        assert k == 2 or np.array_equal(two[k], 1.0 / x[k])


@pytest.mark.gpu
def test_fast_quotients_are_ieee(cuda):
    """sdiv (the mixed and FP64 FMA paths' cell states, and the inversion's setup and result): the
    quotient estimate from the device's reciprocal y, corrected by its remainder, each operation
    rounded once; also with y = the square of the reciprocal of b's root, and from a product."""
    g, geom, conn, aux, _ = make_torus(16, 16, 1)
    dev = Harm(g, geom, conn, aux)
    rng = np.random.default_rng(7)
    n = 4000
    b = np.concatenate([rng.uniform(1.0, 2.0, n // 2), 10.0 ** rng.uniform(-60, 60, n // 2)])
    root, c = np.sqrt(b), rng.uniform(1.0, 9.0, n)
    recip = []
    for v in (b, root, b * c):
        r = cuda.empty(n, dtype=cuda.float64, device="cuda")
        dev.mixed_reciprocal(cuda.from_numpy(v).cuda(), r)
        recip.append(r.cpu().numpy())
    a = rng.uniform(-1.0, 1.0, n) * b * 10.0 ** rng.uniform(-9, 3, n)
    for y in (recip[0], recip[1] * recip[1], recip[2] * c):
        q = a * y
        for k in range(n):
            rem = float(Fraction(a[k]) - Fraction(b[k]) * Fraction(q[k]))
            assert float(Fraction(rem) * Fraction(y[k]) + Fraction(q[k])) == a[k] / b[k], k
