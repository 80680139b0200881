"""A fit solved by t threads rounds the same in every kernel: the first level's,
one per ROI side, and the list kernel and the warp solver that go on with it
past the iteration budget. With the same t before and after, the budget must
not show in the rows, bit for bit."""
import numpy as np
import pytest

import localizer_b200 as L
from tests.test_gpu_fit_routes import _fit, _stack, engine  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [1, 2, 3, 5, 7, 8, 9, 13])
@pytest.mark.parametrize("method", [0, 1, 7])
def test_budget_does_not_show(engine, method, half):  # noqa: F811
    frames, cands = _stack(half, 4200, 77 * half)
    for threads in (1, 4, 8):
        for pivot in (0.0, 1e-2):   # with and without the FP64 pivot escalation's kernels
            kw = dict(threads_per_fit=threads, tail_threads_per_fit=threads, fp64_rerun=-1, pivot_threshold=pivot)
            rows, flags = _fit(engine, frames, cands, method, level0_budget=-1, **kw)
            for budget in (2, 6):
                r, f = _fit(engine, frames, cands, method, level0_budget=budget, **kw)
                np.testing.assert_array_equal(f, flags, err_msg=f"{threads} threads, budget {budget}, pivot {pivot}")
                np.testing.assert_array_equal(r, rows, err_msg=f"{threads} threads, budget {budget}, pivot {pivot}")
