"""The row-major ingest kernel at the sizes where it can go wrong: frames
smaller than a tile, one pixel short of and past tile edges, odd sides (output
rows that start at an odd pixel), single rows and columns, sources and
destinations off their natural alignment, and the count of changed pixels.
Pixels are whole numbers and compared exactly."""
import ctypes as C

import numpy as np
import pytest

import localizer_b200 as L

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 7), (2, 7, 1), (1, 2, 130), (3, 63, 65), (2, 64, 63), (2, 65, 64), (1, 64, 64), (3, 127, 129),
          (2, 128, 66)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", ["uint8", "int16", "uint16", "float32", "float64"])
@pytest.mark.parametrize("shift", [0, 1])
def test_row_major(shape, dtype, shift):
    """shift: the source and the destination start one element further."""
    import torch
    rng = np.random.default_rng(sum(shape))
    x = rng.integers(0, 200, shape).astype(dtype)
    if dtype.startswith("float"):
        x = (x + rng.choice([0.0, 0.25], shape)).astype(dtype)
    elif dtype == "int16":
        x = (x - 100).astype(dtype)
    n, rows, cols = shape
    as_bytes = np.concatenate([np.zeros(x.itemsize * shift, np.uint8), np.frombuffer(x.tobytes(), np.uint8)])
    src = torch.from_numpy(as_bytes).cuda()
    dst = torch.full((x.size + shift + 8,), -1, dtype=torch.int16, device="cuda")
    torch.cuda.synchronize()
    lossy = L.lib().loc_ingest_frames(C.c_void_p(src.data_ptr() + x.itemsize * shift), L.STORAGE_FORMATS[dtype], n, rows,
                                      cols, 1, C.c_void_p(dst.data_ptr() + 2 * shift), C.c_void_p(0))
    got = dst.cpu().numpy().view(np.uint16)
    want = np.clip(np.rint(x.astype(np.float64)), 0, 65535)
    np.testing.assert_array_equal(got[shift:shift + x.size].reshape(n, cols, rows), want.transpose(0, 2, 1))
    assert (got[:shift] == 65535).all() and (got[shift + x.size:] == 65535).all()   # nothing else is written
    assert lossy == int((want != x).sum())
