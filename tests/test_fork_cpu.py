"""A process forks that has made a host call large enough for the copying threads: the child has the library's memory and
none of its threads, and ends like any other."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import ctypes as C, os, sys
import numpy as np
from tests.fake_cuda import wrap_nvfp4
fake = C.CDLL(sys.argv[1])
assert fake.coli_cuda_init((C.c_int * 1)(0), 1)
H, I, rows = 1024, 16, 64
tensors = [(C.c_void_p * 1)(wrap_nvfp4(fake, o, i)) for o, i in ((I, H), (I, H), (H, I))]
x, y = np.zeros((rows, H), np.float32), np.zeros((rows, H), np.float32)  # 256 KB each
def threads():
    return len(os.listdir("/proc/self/task"))
before = threads()
fake.coli_cuda_expert_group_nvfp4(*tensors, (C.c_int * 1)(rows), 1, y.ctypes.data_as(C.c_void_p), x.ctypes.data_as(C.c_void_p))
assert threads() > before or os.cpu_count() < 4
pid = os.fork()
if pid == 0:
    if sys.argv[2] == "call":
        fake.coli_cuda_expert_group_nvfp4(*tensors, (C.c_int * 1)(rows), 1, y.ctypes.data_as(C.c_void_p), x.ctypes.data_as(C.c_void_p))
    if sys.argv[2] == "shutdown":
        fake.coli_cuda_shutdown()
    C.CDLL(None).exit(0)
code = os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1])
assert code == 0, code
fake.coli_cuda_shutdown()
assert threads() == before
C.CDLL(None).exit(0)
"""


@pytest.mark.parametrize("child", ["exit", "call", "shutdown"])
def test_a_forked_child_ends_normally(fake_cuda, child):
    r = subprocess.run([sys.executable, "-c", SCRIPT, fake_cuda._name, child], cwd=ROOT, env={**os.environ, "OPENBLAS_NUM_THREADS": "1"}, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr)
