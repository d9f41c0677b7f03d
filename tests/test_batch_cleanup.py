"""A batch that fails between a round's launch and the wait for it (on the CPU, on a
fake CUDA runtime whose launch of the round's counter kernel fails): the batch's own
stream, with memsets and a kernel in flight on the contexts' memory, is waited for
before any context gives its memory back for another thread to take."""
import fakecuda

BATCH = """
shape = (20, 18, 24)
fields = [np.full(tuple(n + 2 for n in shape), 1e10) for _ in range(3)]
try:
    api.solve_batch(fields, [(1.0, 1.0, 1.0)] * 3, precision=L.PREC_FP32)
    print("ok")
except api.PdfsError as e:
    print("error", e.status)
"""


def test_batch_runs_on_the_fake_runtime():
    text, log = fakecuda.run(BATCH)
    assert text.split() == ["ok"]
    assert any(w[0] == "launch" and "pc_sweep_kernel" in w[1] for w in log)


def test_failed_round_is_waited_for_before_its_memory_is_given_back():
    text, log = fakecuda.run(BATCH, fail="k_add")
    assert text.split() == ["error", "-3"]
    at = next(i for i, w in enumerate(log) if w[0] == "fail")
    stream = log[at][-1]  # the batch's
    assert any(w[0] == "launch" and "pc_sweep_kernel" in w[1] and w[-1] == stream for w in log[:at])
    after = [w for w in log[at + 1:] if w[0] in ("wait", "free", "malloc")]
    assert after[0] == ["wait", stream]
    # every context's stream comes later: destroying it is what gives its memory back
    others = {w[-1] for w in log[:at] if w[0] in ("launch", "copy", "set")} - {stream, "stream0"}
    assert len(others) == 3 and {w[-1] for w in after if w[0] == "wait"} == others | {stream}
