"""Lists longer than the warp solver takes. In a call of some thousand fits all
lists are short enough for it; here most fits outlive the first level and nearly
all are flagged, so that the second level's list, both sets of FP64 re-runs
(short and long, sharing their arrays from both ends) and what their thread
groups leave over are worked on by groups of every size. Rows, flags and
diagnostics must be those of calls that go to the warps alone, bit for bit, and
the same in a second run, whatever warp ran dry first."""
import numpy as np
import pytest
import torch

import localizer_b200 as L
from tests.test_gpu_fit_routes import TEAM_ONLY, _stack

pytestmark = pytest.mark.gpu

N, PART = 12000, 3000


def _fit(engine, frames, cands, method, **kw):
    n = len(cands)
    fd = torch.from_numpy(frames.view(np.int16)).cuda()
    cd = torch.from_numpy(np.ascontiguousarray(cands).view(np.uint8)).cuda()
    out = torch.zeros((n, L.lib().loc_output_columns(method)), dtype=torch.float64, device="cuda")
    flags = torch.zeros(n, dtype=torch.uint8, device="cuda")
    diag = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
    o = L.default_options(rerun_iters=1, rerun_skip_rejected=-1.0, **kw)
    o.d_diag = diag.data_ptr()
    engine.fit_device(fd.data_ptr(), fd.shape[0], fd.shape[2], fd.shape[1], cd.data_ptr(), n, method, 1.5, 1.0,
                      out.data_ptr(), flags.data_ptr(), torch.cuda.current_stream().cuda_stream, o)
    torch.cuda.synchronize()
    return out.cpu().numpy(), flags.cpu().numpy(), diag.cpu().numpy()


# first-level budget, iterations from which a re-run is long, threads of the
# second level, of the short and of the long re-runs, all on one stream
@pytest.mark.parametrize("method,half,budget,long_iters,tail,short,long_,serial", [
    (7, 4, 3, 0, 8, 2, 8, 0), (7, 5, 2, 12, 4, 1, 4, 0), (7, 3, 4, 2, 1, 4, 2, 0), (7, 6, 3, -1, 8, 8, 8, 1),
    (0, 4, 3, 0, 8, 2, 8, 0), (0, 5, 2, 8, 4, 4, 1, 0), (0, 3, 6, 3, 8, 8, 4, 1), (0, 7, 4, -1, 1, 1, 8, 0),
    (1, 4, 2, 0, 8, 2, 8, 0), (1, 2, 3, 2, 4, 4, 2, 1), (5, 4, 3, 6, 8, 2, 4, 0), (7, 1, 3, 0, 8, 2, 8, 0),
    (0, 1, 4, 12, 4, 1, 4, 0), (1, 1, 3, 0, 8, 2, 8, 0)])
def test_long_lists(method, half, budget, long_iters, tail, short, long_, serial):
    frames, cands = _stack(half, N, 31 * half + method)
    kw = dict(level0_budget=budget, long_rerun_iters=long_iters, tail_threads_per_fit=tail,
              rerun_threads_per_fit=short, long_rerun_threads_per_fit=long_)
    eng = L.Engine(0)
    whole = _fit(eng, frames, cands, method, serial_classes=serial, **kw)
    # all but the fits that FP32 left at the iteration cap, which of five
    # parameters in nine pixels are most (3 x 3 ROIs have a lower line)
    assert eng.stats()["fits_fp64_rerun"] > (TEAM_ONLY if half == 1 else 2 * TEAM_ONLY)
    again = _fit(eng, frames, cands, method, serial_classes=serial, **kw)
    parts = [_fit(eng, frames, cands[k:k + PART], method, **kw) for k in range(0, N, PART)]
    eng.close()
    for w, a, p in zip(whole, again, (np.concatenate(x) for x in zip(*parts))):
        np.testing.assert_array_equal(a, w)
        np.testing.assert_array_equal(p, w)
