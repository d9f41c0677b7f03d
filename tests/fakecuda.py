"""Runs a piece of Python on the library's host code with no GPU: a child process with
tests/fake_cudart.c preloaded in the CUDA runtime's place."""
import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
_so = None


def _shim():
    global _so
    if _so is None:
        d = tempfile.mkdtemp(prefix="fake_cudart")
        _so = os.path.join(d, "fake_cudart.so")
        subprocess.run(["gcc", "-O1", "-shared", "-fPIC", os.path.join(HERE, "fake_cudart.c"), "-o", _so, "-lpthread"],
                       check=True)
    return _so


def run(code, memory=None, fail=None, env=None):
    """Runs code (with np, L and api imported); returns its stdout and the runtime's
    log as lists of words.  memory: bytes of the device; fail: part of the name of the
    kernel whose first launch fails; env: more variables."""
    with tempfile.TemporaryDirectory() as d:
        log = os.path.join(d, "log")
        e = dict(os.environ, LD_PRELOAD=_shim(), FAKE_LOG=log, **(env or {}))
        if memory is not None:
            e["FAKE_MEMORY"] = str(int(memory))
        if fail is not None:
            e["FAKE_FAIL"] = fail
        pre = "import sys; sys.path.insert(0, %r)\nimport numpy as np\nfrom pdfs_gb300 import _lib as L, api\n" % ROOT
        r = subprocess.run([sys.executable, "-c", pre + code], env=e, cwd=ROOT, text=True, capture_output=True)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout, [line.split() for line in open(log)]


def copies(code, nbytes):
    """The host data of every copy to the device of nbytes bytes, in order."""
    with tempfile.TemporaryDirectory() as d:
        f = os.path.join(d, "copies")
        run(code, env={"FAKE_COPIES": f, "FAKE_COPY_BYTES": str(nbytes)})
        data = open(f, "rb").read() if os.path.exists(f) else b""
    return [data[i:i + nbytes] for i in range(0, len(data), nbytes)]
