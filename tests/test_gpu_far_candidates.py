"""Candidates far outside the frame, finite but beyond the range of an int:
every method flags them as edge rejects and reads no pixel for them."""
import numpy as np
import pytest

import localizer_b200 as L

EDGE = 1


@pytest.mark.gpu
@pytest.mark.parametrize("method", [0, 1, 5, 6, 7])
def test_far_candidates_are_edge_rejects(method):
    far = [2.0 ** 31 - 3, 2.0 ** 31 + 5, 1e12, 1e300, -(2.0 ** 31) - 5, -1e12, -1e300]
    cands = np.zeros(2 * len(far) + 1, L.CANDIDATE_DTYPE)
    cands["x"] = far + [20.0] * len(far) + [20.0]
    cands["y"] = [20.0] * len(far) + far + [20.0]
    cands["intensity"], cands["background"], cands["half_width"] = 100.0, 10.0, 4
    yy, xx = np.mgrid[0:40, 0:40]
    frames = (10 + 100 * np.exp(-((xx - 20) ** 2 + (yy - 20) ** 2) / 4.5)).round().astype(np.uint16)[None]
    eng = L.Engine(0)
    rows, flags = eng.fit_host(frames, cands, method, 1.5)
    eng.close()
    np.testing.assert_array_equal(flags[:-1], EDGE)
    assert np.isnan(rows[:-1, 1:-2]).all() and (rows[:-1, -2:] == 0).all()
    assert flags[-1] == 0
