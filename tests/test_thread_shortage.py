"""A process that is given no thread more: the planners' work is done by the
calling thread, and a call ends in its result or an error code, not in an
abort."""
import os
import resource
import subprocess
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# The stack limit sets the size of a new thread's stack; this one fits no
# address space, so that no thread can start.
PROGRAM = r'''
import os, resource, sys
if len(sys.argv) == 2:
    resource.setrlimit(resource.RLIMIT_STACK, (1 << 46, resource.RLIM_INFINITY))
    os.execv(sys.executable, [sys.executable, sys.argv[0], sys.argv[1], "limited"])
sys.path[:0] = [sys.argv[1], os.path.join(sys.argv[1], "tests")]
import threading
try:
    threading.Thread(target=int).start()
    print("threads start")
except RuntimeError:
    print("no threads", flush=True)
import ctypes as C
from siminf_gb300 import abi, native
import test_batch_slices as T
# the batch merges its events before it asks for a device
models = [T.seir(50, 20, 10, 1), T.seir(3000, 15, 9000, 2)]
from siminf_gb300.run import run_batch
try:
    run_batch(models, [1, 2], cap_transfers=True)
except Exception as e:
    print("error code", e)
print("alive")
'''


def test_batch_merge_and_plan_without_threads(tmp_path):
    if resource.getrlimit(resource.RLIMIT_STACK)[1] != resource.RLIM_INFINITY:
        pytest.skip("the stack limit cannot be raised")
    path = tmp_path / "shortage.py"
    path.write_text(PROGRAM)
    env = dict(os.environ, OPENBLAS_NUM_THREADS="1", OMP_NUM_THREADS="1", CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, str(path), REPO], capture_output=True, text=True, env=env,
                       timeout=300)
    assert "no threads" in r.stdout, r.stdout + r.stderr
    assert r.returncode == 0, r.stderr
    assert "alive" in r.stdout
