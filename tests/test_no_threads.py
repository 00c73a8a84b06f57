"""Host work goes on where the system starts no more threads: building a plan
in a process whose threads cannot be created (a thread's stack does not fit the
address space it may still have) gives what it gives elsewhere, and does not
abort."""
import os
import resource
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
STACK = 4 << 30
WORK = """
import resource, sys, threading, zlib
import gtopen_b200 as g
from gtopen_b200 import workloads as W
spot = g.Spot(W.flop_spot(g.evaluate7, seed=6, bet=("50", "125"), raise_=("2.5x",), max_raises=2, pot=100, stack=500,
                          frac=(0.01, 0.01)))
assert spot.num_nodes > 1 << 20  # plans of smaller trees are built by one thread
if sys.argv[1] == "none":
    used = int(next(x for x in open("/proc/self/status") if x.startswith("VmSize")).split()[1]) << 10
    resource.setrlimit(resource.RLIMIT_AS, (used + (2 << 30), resource.RLIM_INFINITY))
    try:
        threading.Thread(target=int).start()
    except RuntimeError:
        pass
    else:
        raise SystemExit("threads can be started")
print(spot.num_nodes, *(zlib.crc32(g.shard_visited(spot, 0, 1, use_iso=k > 0).tobytes()) for k in (1, 0)))
"""


def _run(mode):
    env = dict(os.environ, OPENBLAS_NUM_THREADS="1", OMP_NUM_THREADS="1")
    hard = resource.getrlimit(resource.RLIMIT_STACK)[1]
    return subprocess.run([sys.executable, "-c", WORK, mode], cwd=ROOT, env=env, capture_output=True, text=True,
                          timeout=300, preexec_fn=lambda: resource.setrlimit(resource.RLIMIT_STACK, (STACK, hard)))


def test_plan_without_threads():
    want, got = _run("all"), _run("none")
    assert want.returncode == 0, want.stderr
    assert got.returncode == 0, got.stderr
    assert got.stdout == want.stdout
