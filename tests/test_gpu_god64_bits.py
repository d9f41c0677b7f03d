"""The FP64 solvers of the bricks (god64.cuh), reference and fast arithmetic, give the
bits of the plain solvers that columns, pencils and batches run.  Whole sweeps over
spheres; and lone nodes between six frozen neighbours, their minima drawn around the
edges of the solvers' branches: where the one-term solution meets the second minimum,
where the two-term one meets the third (from single units in the last place to some 1e7 of them),
and where the bounds that foretell the third term stop being sure."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (8, 8, 16), (9, 8, 17), (7, 15, 15), (8, 1, 33), (33, 50, 8), (50, 43, 52)]
SPACINGS = [(1.0, 1.0, 1.0), (0.7, 1.3, 0.4), (1.0 / 63, 1.0 / 63, 1.0 / 31), (0.02, 1.0, 3.0)]
PLAIN = [1, 4]  # column tiles: the plain solvers


def sweeps(field, frozen, sp, arith, tile, orderings=range(1, 9)):
    nz, ny, nx = (n - 2 for n in field.shape)
    out = np.empty_like(field)
    with api.Context(nx, ny, nz, sp, freeze=L.FREEZE_MASK, precision=L.PREC_FP64, arith=arith, tile=tile << 8) as c:
        c.load(field, frozen)
        changes = [c.sweep(sn) for sn in orderings]
        c.store(out)
    return out, changes


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sp", SPACINGS)
def test_fast_sweeps_equal_plain_solver(shape, sp):
    w = W.random_spheres(*shape, *sp, 4, 1.5 * sp[0], 9.0 * sp[0], seed=sum(shape))
    w.field[1, 1, 1] = 0.25 * sp[0]
    for frozen in (w.frozen, None):
        a = sweeps(w.field, frozen, sp, L.ARITH_FAST, 6)
        for tile in PLAIN:
            b = sweeps(w.field, frozen, sp, L.ARITH_FAST, tile)
            assert a[0].tobytes() == b[0].tobytes()
            assert a[1] == b[1]


@pytest.mark.parametrize("h", [1e-40, 1e-25, 1e-12, 1e14, 1e25, 1e40])
def test_fast_at_extreme_spacings(h):
    w = W.random_spheres(20, 13, 35, 1.0, 1.0, 1.0, 4, 1.5, 9.0, seed=68)
    f = np.where(w.field < 1e4, w.field * h, 1e4 * h)
    a, b = (sweeps(f, w.frozen, (h, 1.5 * h, 0.5 * h), L.ARITH_FAST, t)[0] for t in (6, 1))
    assert np.array_equal(a, b, equal_nan=True)


def test_fast_on_odd_values():
    r = np.random.default_rng(7)
    f = r.uniform(0.0, 3.0, (37, 22, 19))
    odd = np.array([-1.5, 0.0, -0.0, 5e-324, 1e-300, 1e9, 1e155, 1e300, 1.7e308, np.inf, np.inf, np.nan, 2.0, 2.0])
    pick = r.random(f.shape) < 0.2
    f[pick] = r.choice(odd, pick.sum())
    frozen = (r.random(f.shape) < 0.1).astype(np.uint8)
    a, b = (sweeps(f, frozen, (1.0, 1.0, 1.0), L.ARITH_FAST, t)[0] for t in (6, 1))
    assert np.array_equal(a, b, equal_nan=True)


def lone_nodes(sp, base, seed, k=30):
    """A grid of 3k nodes a side whose free nodes, one in 27, have six frozen
    neighbours of their own."""
    r = np.random.default_rng(seed)
    n = 3 * k
    f = np.full((n + 2,) * 3, 1e6 + base)
    frozen = np.ones(f.shape, np.uint8)
    at = np.stack(np.meshgrid(*[np.arange(2, n, 3)] * 3, indexing="ij"), -1).reshape(-1, 3)  # z, y, x
    frozen[tuple(at.T)] = 0
    m = len(at)
    perm = np.argsort(r.random((m, 3)), 1)  # the axes (x, y, z) by rising minimum
    d = np.asarray(sp)[perm]
    m0 = base * r.random(m)
    kind = r.integers(0, 4, m)
    a = d[:, 0] * np.where(kind == 0, 1.0 + 2.0**-40 * r.integers(-3, 4, m), r.random(m))
    m1 = m0 + a
    w0, w1 = 1 / d[:, 0]**2, 1 / d[:, 1]**2
    root = np.sqrt(np.maximum(w0 + w1 - (m1 - m0)**2 * w0 * w1, 0))
    u2 = m0 + ((m1 - m0) * w1 + root) / (w0 + w1)
    # the third minimum: anywhere; within ulps of u2; where (m2 - m0)^2 w0 + (m2 - m1)^2 w1 is 1 - eps
    eps = 10.0 ** r.uniform(-7, -3, m)
    edge = m0 + ((m1 - m0) * w1 + np.sqrt(np.maximum(root**2 - eps * (w0 + w1), 0))) / (w0 + w1)
    m2 = np.select([kind <= 1, kind == 2], [m1 + (u2 - m1) * 1.5 * r.random(m), u2], edge)
    ulps = np.where(r.random(m) < 0.5, r.integers(-6, 7, m), np.rint(r.choice([-1, 1], m) * 10.0 ** r.uniform(0, 7, m)))
    m2 = np.where(kind == 2, m2 + np.spacing(u2) * ulps, m2)
    mins = np.stack([m0, m1, m2], 1)
    for i in range(3):
        ax = 2 - perm[:, i]  # axis x is the last index
        off = np.zeros((m, 3), int)
        off[np.arange(m), ax] = np.where(r.random(m) < 0.5, 1, -1)
        f[tuple((at + off).T)] = mins[:, i]
    return f, frozen


@pytest.mark.parametrize("arith", [L.ARITH_REFERENCE, L.ARITH_FAST])
@pytest.mark.parametrize("sp", SPACINGS)
@pytest.mark.parametrize("base", [0.0, 1.0, 300.0, 1e5])
def test_lone_nodes_at_the_branches(arith, sp, base):
    f, frozen = lone_nodes(sp, base, int(base) + 1)
    a, b = (sweeps(f, frozen, sp, arith, t, (1,))[0] for t in (6, 1))
    free = frozen == 0
    assert (a[free] < 1e6 + base).all()  # every one updates
    assert a.tobytes() == b.tobytes()


def test_batch_equals_lone_solve_in_fast_arithmetic():
    kw = dict(precision=L.PREC_FP64, arith=L.ARITH_FAST, tol=1e-9)
    ws = [W.random_spheres(*s, 1.0, 1.0, 1.0, 3, 1.5, 8.0, seed=k) for k, s in enumerate([(50, 33, 20), (17, 31, 64)])]
    fields = [w.field.copy() for w in ws]
    st = api.solve_batch(fields, [(1.0, 1.0, 1.0)] * 2, frozen=[w.frozen for w in ws], freeze=L.FREEZE_MASK, **kw)
    for w, f, s in zip(ws, fields, st):
        ref = w.field.copy()
        api.solve(ref, (1.0, 1.0, 1.0), frozen=w.frozen, freeze=L.FREEZE_MASK, fixed_sweeps=s["sweeps_fp64"], **kw)
        assert f.tobytes() == ref.tobytes()
