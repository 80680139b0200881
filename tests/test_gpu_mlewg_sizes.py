"""The warp-per-fit MLEwG kernel at the sizes where its pixel loop can go
wrong (fewer pixels than lanes, one and several chunks of 64 terms, the
largest ROI), against the restated Nelder-Mead minimiser
(oracle/nmsimplex_core.c) driven by a numpy objective in the reference's
operation order.

Both sides run the same FP64 sequence up to the last bit of exp, log and
lgamma. A flipped comparison late in a run ends it at another corner of a
converged simplex (size 1e-2 or the 200-iteration cap), which moves a
position by less than 1e-2 px; the gate is 1e-3 px, as for the golden
fixture, for all but one fit of a case (1 of 24 is the fixture's 0.5 % at the
90 % confidence level)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import localizer_b200 as L

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NM_NMAX = 8


class NmState(C.Structure):
    _fields_ = [("n", C.c_int), ("x1", C.c_double * ((NM_NMAX + 1) * NM_NMAX)), ("y1", C.c_double * (NM_NMAX + 1)),
                ("center", C.c_double * NM_NMAX), ("ws", C.c_double * (4 * NM_NMAX)), ("S2", C.c_double)]


@pytest.fixture(scope="module")
def nm(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("nm") / "nm.so")
    subprocess.run(["gcc", "-O2", "-fPIC", "-fno-fast-math", "-ffp-contract=off", "-std=c11", "-shared", "-o", so,
                    os.path.join(ROOT, "oracle", "nmsimplex_core.c"), "-lm"], check=True)
    return C.CDLL(so)


def _oracle_fit(nm, roi, xo, yo, cand, w0):
    """(x, y) and the iteration count of the reference's minimisation."""
    from scipy.special import gammaln
    s = roi.shape[0]
    d = roi.astype(np.float64).ravel()
    x = np.tile(xo + np.arange(s, dtype=np.float64), s)
    y = np.repeat(yo + np.arange(s, dtype=np.float64), s)
    lg = gammaln(d + 1.0)
    fn_t = C.CFUNCTYPE(C.c_double, C.POINTER(C.c_double), C.c_void_p)

    def f(p, _):
        with np.errstate(all="ignore"):
            e = p[4] / (2 * np.pi * p[2] * p[2]) * np.exp(-((x - p[0]) * (x - p[0]) + (y - p[1]) * (y - p[1]))
                                                          / p[2] / p[2]) + p[3]
            return float(-1.0 * np.cumsum(-e + d * np.log(e) - lg)[-1])   # cumsum adds in order
    cb = fn_t(f)
    v = (C.c_double * 5)(cand["x"], cand["y"], w0, cand["background"], cand["intensity"] * 2 * np.pi * w0 * w0)
    st, size, fv, step = NmState(), C.c_double(), C.c_double(), (C.c_double * 5)(1, 1, 1, 1, 1)
    assert nm.nm_set(C.byref(st), 5, cb, None, v, step, C.byref(size)) == 0
    it = 0
    while it < 200:
        it += 1
        if nm.nm_iterate(C.byref(st), cb, None, v, C.byref(size), C.byref(fv)) or size.value < 1e-2:
            break
    return v[0], v[1], it


@pytest.mark.parametrize("r", [2, 3, 4, 8, 16])
def test_mlewg_roi_sizes(nm, r):
    rng = np.random.default_rng(40 + r)
    n, side, w0 = 24, 2 * r + 9, 1.4
    yy, xx = np.mgrid[0:side, 0:side]
    frames, cands = np.empty((n, side, side), np.uint16), np.zeros(n, L.CANDIDATE_DTYPE)
    for k in range(n):
        cx, cy = side / 2 + rng.uniform(-1, 1, 2)
        lam = 60 + 700 * np.exp(-((xx - cx) ** 2 + (yy - cy) ** 2) / (2 * 1.4 ** 2))
        frames[k] = rng.poisson(lam)
        cands[k] = (round(cx), round(cy), float(frames[k].max()) - 60.0, 60.0, k, r)
    eng = L.Engine(0)
    rows, flags = eng.fit_host(frames, cands, L.METHOD_MLEWG, w0)
    bounded, bflags = eng.fit_host(frames, cands, L.METHOD_MLEWG, w0, options=L.default_options(max_half_width=r))
    eng.close()
    np.testing.assert_array_equal(rows, bounded)     # the half-width promise changes the launch only
    np.testing.assert_array_equal(flags, bflags)
    off = 0
    for k in range(n):
        xo, yo = int(np.floor(cands[k]["x"] - r)), int(np.floor(cands[k]["y"] - r))
        x, y, it = _oracle_fit(nm, frames[k, yo:yo + 2 * r + 1, xo:xo + 2 * r + 1], xo, yo, cands[k], w0)
        if flags[k] == 0 and not (rows[k, -2] == it and max(abs(rows[k, 3] - x), abs(rows[k, 4] - y)) < 1e-3):
            off += 1
    assert (flags == 0).sum() >= n // 2 and off <= 1, (off, flags)
