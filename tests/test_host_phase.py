"""The threaded host phase where the system starts no thread: the result comes out all the same,
and the process goes on."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CHILD = r"""
import ctypes as C, os, resource, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from cuphu_b200._lib import lib
fn = lib()._ZN5cuphu18compute_host_phaseEPKfS1_S1_mPf   # cuphu::compute_host_phase
fn.restype = None
fn.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p]
n = 1 << 16
rng = np.random.default_rng(2)
ig = rng.normal(size=2 * n).astype(np.float32)

def phase(threads):
    os.environ["CUPHU_HOST_THREADS"] = threads
    C.CDLL(None).setenv(b"CUPHU_HOST_THREADS", threads.encode(), 1)
    out = np.full(n, np.nan, np.float32)
    fn(ig.ctypes.data, None, None, n, out.ctypes.data)
    return out

want = phase("1")
out = np.empty(n, np.float32)
# no room for a thread's stack any more
with open("/proc/self/statm") as f:
    size = int(f.read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (size + (3 << 20), resource.RLIM_INFINITY))
got = phase("4")
assert np.array_equal(got, want)
print("same")
"""


def test_phase_without_threads():
    r = subprocess.run([sys.executable, "-c", _CHILD, ROOT], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, (r.returncode, r.stdout, r.stderr)
