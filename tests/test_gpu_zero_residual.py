"""Fits whose residual is exactly zero end at the iteration cap in their first
iteration when the stopping test cannot hold (a zero tolerance). With
rerun_capped they are all solved again in FP64, as long ones, more of them
than the warp solver takes before the thread groups work on a list; their rows
must be those of calls small enough for the warps alone."""
import numpy as np
import pytest

import localizer_b200 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [0, 1, 7])
def test_zero_residual_fits_are_solved_again(method):
    n, part = 9000, 3000
    frames = np.zeros((1, 32, 32), np.uint16)
    cands = np.zeros(n, L.CANDIDATE_DTYPE)
    cands["x"], cands["y"] = 16.0, 16.0
    cands["half_width"] = 3
    eng = L.Engine(0)
    opts = dict(epsabs=0.0, rerun_capped=1, host_roi_mode=-1, rerun_skip_rejected=-1.0)
    rows, flags = eng.fit_host(frames, cands, method, 1.5, options=L.default_options(**opts))
    st = eng.stats()
    r, f = eng.fit_host(frames, cands[:part], method, 1.5, options=L.default_options(**opts))
    eng.close()
    assert (r[:, -2] == L.default_options().max_iter).all()   # the cap
    for k in range(0, n, part):
        np.testing.assert_array_equal(flags[k:k + part], f)
        np.testing.assert_array_equal(rows[k:k + part], r)
    assert st["fits_fp64_rerun"] == n, st
