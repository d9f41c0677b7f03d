"""The replace-update's cap bounds (k_block_capmin in solver.cu): per 8^3 block the
smallest input of the nodes the sweeps update, +inf where every node is frozen, and
the same rounded down to float -- exactly, at widths that leave 1 to 4 blocks to the
last CTA of a row, with fully frozen blocks beside blocks of small values."""
import ctypes as C

import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (8, 8, 8), (9, 7, 17), (31, 3, 2), (33, 8, 17), (57, 20, 9), (127, 2, 9), (130, 25, 33)]


def block_min(v, use, nb):
    nbz, nby, nbx = nb
    p = np.full((8 * nbz, 8 * nby, 8 * nbx), np.inf)
    nz, ny, nx = v.shape
    p[:nz, :ny, :nx] = np.where(use, v, np.inf)
    return p.reshape(nbz, 8, nby, 8, nbx, 8).min(axis=(1, 3, 5))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("masked", [False, True])
def test_block_minima(shape, masked):
    nx, ny, nz = shape
    r = np.random.default_rng(sum(shape))
    f = r.uniform(0.5, 9.0, (nz + 2, ny + 2, nx + 2))
    f[1:-1, 1:-1, 1:-1] += 10.0 * (np.arange(nx) // 8 % 3)  # neighbours far apart, the smaller ones first
    frozen = (r.random(f.shape) < 0.1).astype(np.uint8)
    frozen[1:-1, 1:-1, 9:17] = 1  # the second block of a row frozen whole
    i = (slice(1, -1),) * 3
    lib = L.load()
    with api.Context(nx, ny, nz, (1.0, 1.0, 1.0), freeze=L.FREEZE_MASK if masked else L.FREEZE_NONE,
                     precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR) as c:
        c.load(f, frozen if masked else None)
        nb = c.blocks()[::-1]
        c64, c32 = np.zeros(nb), np.zeros(nb, np.float32)
        lib.pdfs_test_caps.argtypes = [C.c_void_p] * 3
        assert lib.pdfs_test_caps(c.h, c64.ctypes.data, c32.ctypes.data) == L.PDFS_OK
    want = block_min(f[i], frozen[i] == 0 if masked else np.ones(f[i].shape, bool), nb)
    down = want.astype(np.float32)
    down = np.where(down > want, np.nextafter(down, np.float32(-np.inf)), down)
    assert np.array_equal(c64, want)
    assert np.array_equal(c32, down)
