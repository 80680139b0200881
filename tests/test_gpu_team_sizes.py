"""The warp solver at the ROI sides that tests/test_gpu_fit_routes.py leaves
out: the smallest, the two others with kernels of their own, one without, and
with them the chunks of whole rows that fill a warp's 64 records almost (63 of
3 x 3 ROIs), from whose end the solver reads ahead. A candidate's row must not
depend on the size of its call, bit for bit."""
import numpy as np
import pytest

import localizer_b200 as L
from tests.test_gpu_fit_routes import TEAM_ONLY, _fit, _stack, engine  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [1, 6, 7, 12])
@pytest.mark.parametrize("method", [0, 1, 7])
@pytest.mark.parametrize("precision", [0, 1])
def test_rows_do_not_depend_on_call_size(engine, method, half, precision):  # noqa: F811
    frames, cands = _stack(half, 4200, 500 * half + method)
    rows, flags = _fit(engine, frames, cands, method, precision=precision)
    for lo, m in ((0, 1), (100, 700), (0, TEAM_ONLY)):
        r, f = _fit(engine, frames, cands[lo:lo + m], method, precision=precision)
        np.testing.assert_array_equal(f, flags[lo:lo + m])
        np.testing.assert_array_equal(r, rows[lo:lo + m])
