"""pdfs_ctx_orderings on a context whose FP32 field no phase has written (FP64 sweeps of an
FP32 + polish context): no node has a value, so no block names an ordering -- also where
the context's memory was another's, with distances in its FP32 field."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(40, 33, 50), (17, 64, 9)])
def test_no_orderings_without_an_fp32_field(shape):
    w = W.random_spheres(*shape, 1.0, 1.0, 1.0, 3, 2.0, 8.0, seed=2)
    kw = dict(freeze=L.FREEZE_MASK, precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR, tol=1e-5)
    with api.Context(*shape, (1.0, 1.0, 1.0), **kw) as c:
        c.load(w.field, w.frozen)
        c.run()
        ran = c.orderings()
    assert ran.any()
    with api.Context(*shape, (1.0, 1.0, 1.0), **kw) as c:  # on the same memory
        c.load(w.field, w.frozen)
        c.sweep(1)
        assert not c.orderings().any()
        c.run()
        assert np.array_equal(c.orderings(), ran)
