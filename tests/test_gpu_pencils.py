"""The pencils' lone sweeps (pair and mixed arithmetic, both updates, both spacing kinds),
which run on large grids: a test hook asks for them on small ones, and the bits are the
bricks' after each of the 8 orderings and at the end of a polish -- at one node past a
pencil, one short of it, one pencil, several, long and short columns."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

HOOK = "PDFS_TEST_PLAIN_PENCILS"
SHAPES = [(1, 1, 1), (16, 16, 16), (17, 16, 33), (15, 31, 31), (16, 1, 65), (33, 50, 8), (50, 43, 52), (97, 33, 64)]
SPACINGS = [(1.0, 1.0, 1.0), (0.7, 1.0, 0.5)]
ARITH = [L.ARITH_PAIR, L.ARITH_MIXED]


def field(shape, sp):
    w = W.random_spheres(*shape, *sp, 4, 1.5, 9.0, seed=sum(shape))
    w.field[1, 1, 1] = 0.25
    return w


def both(monkeypatch, f):
    a = f()
    monkeypatch.setenv(HOOK, "1")
    b = f()
    monkeypatch.delenv(HOOK)
    return a, b


@pytest.mark.parametrize("arith", ARITH)
@pytest.mark.parametrize("sp", SPACINGS)
@pytest.mark.parametrize("shape", SHAPES)
def test_sweeps_equal_bricks(shape, sp, arith, monkeypatch):
    w = field(shape, sp)
    for frozen in (w.frozen, None):

        def sweeps():
            out = np.empty_like(w.field)
            with api.Context(w.nx, w.ny, w.nz, sp, freeze=L.FREEZE_MASK, precision=L.PREC_FP64, arith=arith) as c:
                c.load(w.field, frozen)
                changes = [c.sweep(sn) for sn in range(1, 9)]
                c.store(out)
            return out.tobytes(), changes

        a, b = both(monkeypatch, sweeps)
        assert a[0] == b[0]
        assert a[1] == pytest.approx(b[1], rel=1e-6)  # the change of a node, in either kernel's rounding


@pytest.mark.parametrize("arith", ARITH)
@pytest.mark.parametrize("sp", SPACINGS)
@pytest.mark.parametrize("shape", [(17, 9, 33), (50, 43, 52), (40, 23, 70)])
def test_polish_equals_bricks(shape, sp, arith, monkeypatch):
    w = W.random_spheres(*shape, *sp, 3, 2.0, 8.0, seed=sum(shape))

    def solve():
        a = w.field.copy()
        st = api.solve(a, sp, frozen=w.frozen, freeze=L.FREEZE_MASK, precision=L.PREC_FP32_POLISH64, arith=arith,
                       tol=1e-5)
        return a.tobytes(), st["sweeps_fp64"]

    a, b = both(monkeypatch, solve)
    assert a == b


def test_bounded_wait_times_out(monkeypatch):
    w = field((50, 43, 52), (1.0, 1.0, 1.0))
    monkeypatch.setenv(HOOK, "1")
    monkeypatch.setenv("PDFS_TEST_POISON_COLUMN", "0")
    with api.Context(w.nx, w.ny, w.nz, (1.0, 1.0, 1.0), precision=L.PREC_FP64, arith=L.ARITH_PAIR, wait_ms=50) as c:
        c.load(w.field)
        with pytest.raises(api.PdfsError) as e:
            c.sweep(1)
        assert e.value.status == L.PDFS_ERR_TIMEOUT
