"""How the host waits for the plain form's rounds (Engine::RunWindows in
beam_gb300/csrc/merge.cu): as the process has asked the driver to wait."""

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

# The flag is set before the context exists, so each form is a process of its own.
CHILD = """
import ctypes, sys, time
sys.path[:0] = [{root!r}]
cuda = ctypes.CDLL("libcuda.so.1")
assert cuda.cuInit(0) == 0
assert cuda.cuDevicePrimaryCtxSetFlags_v2(0, {flag}) == 0
from beam_gb300 import Engine, Graph, partition_hash
g = Graph.generate("rmat:scale=19,ef=16,a=0.57,b=0.19,c=0.19,seed=5")
with Engine(g, ea_use_threshold=True, group_batch_size=1024) as e:
    e.run(1)
    e.reset()
    wall, cpu = time.perf_counter(), time.process_time()
    e.run(2)
    wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
    print(cpu / wall, partition_hash(e.partition()[0]))
"""


def run(flag):
    out = subprocess.run([sys.executable, "-c", CHILD.format(root=str(ROOT), flag=flag)], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    share, labels = out.stdout.split()
    return float(share), labels


def test_blocking_waits_leave_the_core():
    """CU_CTX_SCHED_BLOCKING_SYNC: the launches of a round are some 30 us of the
    host's time, its kernels a millisecond and more on this graph, so the run uses
    less than half of a core; a spin would use all of it."""
    share, labels = run(4)
    assert share < 0.5
    for flag in (0, 1, 2):  # automatic, spin, yield: the same rounds
        assert run(flag)[1] == labels
