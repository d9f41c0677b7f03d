"""The route of plain pair and mixed sweeps (host code on a fake CUDA runtime, no GPU):
the hook that test_gpu_pencils.py sets brings small grids to the pencil kernel's lone
instances -- each of the eight -- and without it they run bricks."""
import re

import pytest

import fakecuda
from pdfs_gb300 import _lib as L

SWEEP = """
kw = %r
f = np.full((26, 22, 18), 1e10)
with api.Context(16, 20, 24, %r, max_sweeps=16, **kw) as c:
    c.load(f)
    c.run()
"""


@pytest.mark.parametrize("arith", [L.ARITH_PAIR, L.ARITH_MIXED])
@pytest.mark.parametrize("sp", [(1.0, 1.0, 1.0), (0.7, 1.0, 0.5)])
@pytest.mark.parametrize("prec", [L.PREC_FP64, L.PREC_FP32_POLISH64])
def test_hook_reaches_every_pencil_instance(prec, sp, arith):
    code = SWEEP % (dict(precision=prec, arith=arith), sp)
    for env in ({}, {"PDFS_TEST_PLAIN_PENCILS": "1"}):
        _, log = fakecuda.run(code, env=env)
        pencils = [w[1] for w in log if w[0] == "launch" and "pc_sweep_kernel" in w[1]]
        assert bool(pencils) == bool(env)
        for n in pencils:  # <double, MODE, ARITH, ISO, BATCH>
            mode, ar, iso, batch = re.search(r"pc_sweep_kernelIdLi(\d)ELi(\d)ELb(\d)ELb(\d)E", n).groups()
            assert (int(mode), int(ar), int(iso), int(batch)) == (int(prec == L.PREC_FP32_POLISH64), int(arith),
                                                                  int(sp[0] == sp[1]), 0)
