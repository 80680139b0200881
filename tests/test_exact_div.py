"""div_by of csrc/loc_div.h against the division it replaces, on the host: equal
bits wherever its two range checks let it run, for one division and for two in
a row, over random operands and the ends of the ranges."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "loc_div.h"
extern "C" long check(const double *a, const double *b, long n, long *used)
{
    long bad = 0, k = 0;
    for (long i = 0; i < n; ++i) {
        if (!locb::in_range(a[i]) || !locb::div_fast(b[i])) continue;
        ++k;
        const double inv = 1.0 / b[i], q = locb::div_by(a[i], b[i], inv);
        bad += q != a[i] / b[i] || locb::div_by(q, b[i], inv) != a[i] / b[i] / b[i];
    }
    *used = k;
    return bad;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "localizer_b200", "csrc"), "-o", str(d / "t.so"), str(d / "t.cpp")], check=True)
    lib = C.CDLL(str(d / "t.so"))
    lib.check.argtypes = [C.c_void_p, C.c_void_p, C.c_long, C.c_void_p]
    lib.check.restype = C.c_long

    def run(a, b):
        a, b = (np.ascontiguousarray(x, np.float64) for x in (a, b))
        used = C.c_long()
        return lib.check(a.ctypes.data, b.ctypes.data, len(a), C.byref(used)), used.value
    return run


def _mantissas(rng, n):
    """Random ones, and among them short ones, all ones and their neighbours."""
    m = 1.0 + rng.random(n)
    few = rng.integers(0, 6, n)
    m = np.where(few == 0, 1.0 + np.floor(rng.random(n) * 64) / 64, m)
    m = np.where(few == 1, np.nextafter(2.0, 0), m)
    m = np.where(few == 2, np.nextafter(1.0 + np.floor(rng.random(n) * 8) / 8, 4), m)
    return m * rng.choice([-1.0, 1.0], n)


@pytest.mark.parametrize("ea,eb", [(12, 3), (299, 99), (305, 104)])
def test_equals_the_division(check, ea, eb):
    rng = np.random.default_rng(ea)
    n = 1_000_000
    a = _mantissas(rng, n) * np.exp2(rng.integers(-ea, ea + 1, n).astype(float))
    b = _mantissas(rng, n) * np.exp2(rng.integers(-eb, eb + 1, n).astype(float))
    # quotients next to a half-way case: a the rounded product of b and a short mantissa
    a[::3] = (b * _mantissas(rng, n))[::3]
    bad, used = check(a, b)
    assert bad == 0 and used > 0.9 * n


def test_ends_of_the_ranges(check):
    a = np.array([s * v for v in (2.0 ** -300, np.nextafter(2.0 ** -300, 1), 1.0, np.nextafter(2.0 ** 300, 1), 2.0 ** 300,
                                  0.0, np.inf, np.nan, 5e-324) for s in (1, -1)])
    b = np.array([2.0 ** -100, np.nextafter(2.0 ** -100, 1), np.nextafter(1.0, 0), 1.5, np.nextafter(2.0 ** 100, 1),
                  2.0 ** 100, 0.0, np.inf, np.nan])
    aa, bb = (x.ravel() for x in np.meshgrid(a, b))
    bad, used = check(aa, bb)
    assert bad == 0 and used == 6 * 4
