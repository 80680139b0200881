"""The filtered GLRT kernel and the run-based grouping at the sizes where they
can go wrong, against the host finder: every window side with its own
instantiation and the general kernel above them, frames smaller than a tile,
one pixel short of and past tile and word boundaries, frames whose window
statistics defeat the FP32 estimate (bright offsets, saturated blocks, a
nearly constant frame), and frames with more runs than the shared run table
holds. Candidates are whole records compared bit for bit."""
import numpy as np
import pytest

import localizer_b200 as L

pytestmark = pytest.mark.gpu


def _check(frames, pfa, width):
    import torch
    host = L.find_candidates(frames, pfa, width)
    raw, n = L.find_candidates_device(torch.from_numpy(frames.view(np.int16)).cuda(), pfa, width)
    assert n == len(host)
    np.testing.assert_array_equal(raw.cpu().numpy(), np.frombuffer(host.tobytes(), np.uint8))
    return n


def _spots(rng, n, cols, rows, bg, count, amp, sigma):
    lam = np.full((n, cols, rows), float(bg))
    yy, xx = np.mgrid[0:cols, 0:rows]
    for f in range(n):
        for _ in range(count):
            x, y = rng.uniform(0, rows), rng.uniform(0, cols)
            lam[f] += amp * np.exp(-((xx - x) ** 2 + (yy - y) ** 2) / (2 * sigma ** 2))
    return np.clip(rng.poisson(lam), 0, 65535).astype(np.uint16)


@pytest.mark.parametrize("width", [0.2, 0.7, 1.2, 1.5, 2.1, 2.6, 3.2, 3.3, 5.0])
def test_window_sides(width):
    """Window sides 1, 3, 5, 7, 9, 11, 13 (own kernels from 3), 15 and 21."""
    rng = np.random.default_rng(int(width * 10))
    frames = _spots(rng, 3, 91, 150, 80, 25, 500, max(width, 0.8))
    found = _check(frames, 30.0, width)
    assert found > 0 or width < 0.5


@pytest.mark.parametrize("cols,rows", [(9, 9), (10, 11), (23, 31), (88, 128), (89, 129), (177, 257), (33, 1000)])
def test_frame_sides(cols, rows):
    rng = np.random.default_rng(cols * rows)
    _check(_spots(rng, 4, cols, rows, 100, 1 + cols * rows // 400, 600, 1.4), 30.0, 1.5)


def test_hard_statistics():
    rng = np.random.default_rng(3)
    f = rng.poisson(100, size=(8, 96, 140)).astype(np.uint16)
    f[0] = 65535                                                    # constant, saturated
    f[1] = 40000 + rng.integers(0, 2, size=f[1].shape)              # nearly constant on an offset
    f[2, 40:50, 40:50] = 65535                                      # saturated block in noise
    f[3] = 0
    f[3, 30, 30] = 1                                                # one count
    f[4, :, 70:] += 30000                                           # a step far above the tile's background
    f[5] = rng.integers(0, 65536, size=f[5].shape)                  # full range noise
    f[6, ::7, ::7] = 60000                                          # hot pixels
    for pfa in (0.01, 1.0, 30.0, 300.0):
        _check(f, pfa, 1.5)


def test_many_runs():
    """Noise at a low threshold: more runs per frame than the shared table,
    more particles than the first guess of the particle table."""
    rng = np.random.default_rng(9)
    frames = rng.poisson(100, size=(3, 400, 420)).astype(np.uint16)
    assert _check(frames, 2.0, 0.7) > 4000
