"""The timestep on streams of the caller's: the legacy default stream (plain launches) and a stream of
another library's (each kernel set up while the one before it runs) give the oracle's bits, beside
work of the caller's on the same stream."""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys
sys.path[:0] = [{pkg!r}, {tests!r}]
import numpy as np, torch, tinymd
from conftest import ORACLE_LIB
from helpers import make_sim
lib, ora = tinymd.load(), tinymd.open_library(ORACLE_LIB)
stream = {stream}
lib.md_set_stream(ctypes.c_void_p(stream.cuda_stream if stream else 0))
a = torch.zeros(1 << 22, device="cuda")
states = []
for l in (lib, ora):
    sim = make_sim(l, cells=(9, 8, 7), setup_lib=lib, reneigh=5)
    for k in range(12):
        if l is lib:
            with torch.cuda.stream(stream or torch.cuda.default_stream()):
                a.add_(1.0)
        sim.step(0.005, 2)
    states.append(tinymd.full_state(l))
    sim.close()
for x, y in zip(*states):
    np.testing.assert_array_equal(x, y)
assert float(a.min()) == float(a.max()) == 12.0
tinymd.check(lib)
print("same")
"""


@pytest.mark.parametrize("stream", ["None", "torch.cuda.Stream()"])
def test_callers_streams(product, oracle, cuda_device, stream):
    script = SCRIPT.format(pkg=PKG, tests=os.path.join(ROOT, "tests"), stream=stream)
    r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("handle", [1, 2])
def test_default_stream_handles(product, oracle, cuda_device, handle):
    """The legacy and per-thread default streams by their handles."""
    script = SCRIPT.format(pkg=PKG, tests=os.path.join(ROOT, "tests"), stream="None").replace(
        "stream.cuda_stream if stream else 0", str(handle)).replace("a.add_(1.0)", "a.add_(1.0); torch.cuda.synchronize()")
    r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr


def test_rebuild_behind_a_long_queue(product, oracle, cuda_device):
    """The ghost count and the list status that the host polls for come late: over a second of the
    caller's work on the same stream is ahead of every rebuild's kernels in the first steps."""
    script = SCRIPT.format(pkg=PKG, tests=os.path.join(ROOT, "tests"), stream="torch.cuda.Stream()").replace(
        "a.add_(1.0)", "a.add_(1.0); k < 3 and torch.cuda._sleep(int(1.6e9))")
    r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
