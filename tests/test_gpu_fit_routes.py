"""The solver's routes give one answer. A fit may be solved by one thread, be
suspended and finished by a group of threads or by a warp, or be solved by a
warp from the start, depending on how many fits its call holds; all routes
compute the same sums in the same order, so rows, flags and diagnostics of a
candidate must not depend on the size of its call, bit for bit. Sizes lie on
both sides of the line below which a call goes to the warps alone, and the ROI
half-widths are the smallest, the ones whose rows the compiler treats apart,
and the largest."""
import numpy as np
import pytest

import localizer_b200 as L

pytestmark = pytest.mark.gpu

TEAM_ONLY = 3552


@pytest.fixture(scope="module")
def engine():
    e = L.Engine(0)
    yield e
    e.close()


def _stack(half, n, seed):
    """n candidates on frames of isolated, elongated, partly dim spots; a few
    candidates point at empty background, whose fits run long."""
    rng = np.random.default_rng(seed)
    size, per = 160, 24
    n_frames = -(-n // per)
    yy, xx = np.mgrid[0:size, 0:size]
    frames = np.empty((n_frames, size, size), np.uint16)
    cands = np.zeros(n_frames * per, L.CANDIDATE_DTYPE)
    for f in range(min(n_frames, 40)):
        lam = np.full((size, size), 90.0)
        for k in range(per):
            x, y = rng.uniform(half + 2, size - half - 3, 2)
            sx, sy = rng.uniform(1.0, 2.2, 2)
            amp = rng.choice([0.0, 25.0, 120.0, 600.0])
            lam += amp * np.exp(-((xx - x) ** 2 / (2 * sx * sx) + (yy - y) ** 2 / (2 * sy * sy)))
            c = cands[f * per + k]
            c["x"], c["y"] = np.round(x), np.round(y)
            c["intensity"], c["background"], c["half_width"] = max(amp, 20.0) * 12.0, 90.0, half
        frames[f] = rng.poisson(lam)
    for f in range(40, n_frames):   # the rest repeats these frames
        frames[f] = frames[f % 40]
        cands[f * per:(f + 1) * per] = cands[(f % 40) * per:(f % 40 + 1) * per]
    cands["frame"] = np.repeat(np.arange(n_frames), per)
    return frames, cands[:n]


def _fit(engine, frames, cands, method, **kw):
    return engine.fit_host(frames, cands, method, 1.5, options=L.default_options(host_roi_mode=-1, **kw))


@pytest.mark.parametrize("half", [2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("method", [0, 1, 5, 7])
@pytest.mark.parametrize("precision", [0, 1])
def test_rows_do_not_depend_on_call_size(engine, method, half, precision):
    n = 4200
    frames, cands = _stack(half, n, 1000 * half + method)
    rows, flags = _fit(engine, frames, cands, method, precision=precision)
    assert (flags == 0).any()
    for lo, m in ((0, 1), (5, 3), (100, 700), (0, TEAM_ONLY), (0, TEAM_ONLY + 1)):
        r, f = _fit(engine, frames, cands[lo:lo + m], method, precision=precision)
        np.testing.assert_array_equal(f, flags[lo:lo + m])
        np.testing.assert_array_equal(r, rows[lo:lo + m])


@pytest.mark.parametrize("method", [0, 7])
@pytest.mark.parametrize("precision", [0, 1])
def test_mixed_half_widths(engine, method, precision):
    """ROIs of every size in one call: warps whose lanes hold different sizes,
    groups without room for the largest, and the cap on the half-width."""
    n = 4200
    frames, cands = _stack(16, n, 77 + method)
    cands["half_width"] = np.random.default_rng(3).integers(2, 17, n)
    rows, flags = _fit(engine, frames, cands, method, precision=precision, max_half_width=16)
    for lo, m in ((0, 64), (640, TEAM_ONLY)):
        r, f = _fit(engine, frames, cands[lo:lo + m], method, precision=precision)
        np.testing.assert_array_equal(f, flags[lo:lo + m])
        np.testing.assert_array_equal(r, rows[lo:lo + m])


@pytest.mark.parametrize("kw", [dict(fp64_rerun=-1), dict(rerun_iters=-1, long_rerun_iters=-1), dict(max_iter=7),
                                dict(pivot_threshold=1e-2), dict(level0_budget=-1)])
def test_options_on_both_routes(engine, kw):
    n = 4200
    frames, cands = _stack(5, n, 5)
    rows, flags = _fit(engine, frames, cands, 7, **kw)
    r, f = _fit(engine, frames, cands[:900], 7, **kw)
    np.testing.assert_array_equal(f, flags[:900])
    np.testing.assert_array_equal(r, rows[:900])


def test_threads_with_other_sizes():
    """Two host threads, each with its own engine, fit ROIs of the smallest and
    the largest size at the same time: the launches share their kernels."""
    import threading
    work = {half: _stack(half, n, half) for half, n in ((2, 4200), (16, 700))}
    want, got, errors = {}, {}, []
    engines = {half: L.Engine(0) for half in work}
    for half, (frames, cands) in work.items():
        want[half] = _fit(engines[half], frames, cands, 7)

    def run(half):
        try:
            for _ in range(20):
                got[half] = _fit(engines[half], *work[half], 7)
        except Exception as e:   # shown by the main thread
            errors.append((half, e))

    threads = [threading.Thread(target=run, args=(half,)) for half in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for half in work:
        np.testing.assert_array_equal(got[half][1], want[half][1])
        np.testing.assert_array_equal(got[half][0], want[half][0])
        engines[half].close()
