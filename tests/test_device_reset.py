"""A program that resets the device (cudaDeviceReset) between solves: the streams, events,
pinned blocks and device memory that idle contexts had left in the library's pools are
gone with the old context, and the next solve takes none of them (host code on a fake CUDA
runtime, which logs every use of a stream or address from before the reset)."""
import fakecuda

SOLVES = """
import ctypes as C
def solve(n, **kw):
    f = np.full((n + 2, n + 2, n + 2), 1e10)
    api.solve(f, (1.0, 1.0, 1.0), max_sweeps=16, **kw)
def everything():
    for n in (20, 40):
        solve(n)
        solve(n, precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR, scheduler=L.SCHED_OCTANT)
    api.solve_batch([np.full((22, 22, 22), 1e10) for _ in range(3)], [(1.0, 1.0, 1.0)] * 3, precision=L.PREC_FP32)
everything()
%s
C.CDLL(None).cudaDeviceReset()
%s
solve(60)
everything()
api.release_cached(0)
print("ok")
"""


def run(before="", after=""):
    text, log = fakecuda.run(SOLVES % (before, after))
    assert [w for w in log if w[0] == "reset"]
    return text.split(), [w for w in log if w[0] == "stale"]


def test_solves_after_a_reset():
    assert run() == (["ok"], [])


def test_pools_emptied_after_a_reset():
    assert run(after="api.release_cached(0)") == (["ok"], [])


def test_context_that_outlives_a_reset():
    """Destroying it gives nothing back to the pools."""
    assert run("c = api.Context(30, 30, 30, (1.0, 1.0, 1.0))", "c.close()") == (["ok"], [])
