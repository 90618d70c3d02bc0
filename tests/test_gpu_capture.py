"""Stream-ordered entry points under stream capture: a capture whose first call is also the
library's first in the process, and one after a call that already made the scratch."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CAPTURE = r"""
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import torch
from cuphu_b200._lib import check, default_params, lib
warm = sys.argv[2] == "warm"
nr, nc = 300, 400
g = torch.Generator(device="cuda")
g.manual_seed(7)
ph, corr = (torch.rand((nr, nc), generator=g, device="cuda") for _ in range(2))
ph *= 6.2
unw = ph + 6.0
fixed = unw.clone()
costs = torch.zeros(((nr - 1) * nc + nr * (nc - 1), 2), dtype=torch.int16, device="cuda")
p = default_params()
torch.cuda.synchronize()

def calls():
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    fixed.copy_(unw)
    check(lib().cuphu_build_costs_device(C.c_void_p(ph.data_ptr()), C.c_void_p(corr.data_ptr()),
                                         None, nr, nc, 0, C.byref(p), C.c_void_p(costs.data_ptr()),
                                         None, s))
    check(lib().cuphu_fix_cycle_spikes_device(C.c_void_p(fixed.data_ptr()), None, nr, nc, s))

if warm:
    calls()
    torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    calls()
costs.zero_()
fixed.zero_()
graph.replay()
torch.cuda.synchronize()
got = costs.clone(), fixed.clone()
calls()
torch.cuda.synchronize()
assert bool((costs != 0).any())
assert torch.equal(got[0], costs) and torch.equal(got[1], fixed)
print("same")
"""


@pytest.mark.parametrize("start", ["first", "warm"])
def test_captured_calls_replay(torch_cuda, start):
    r = subprocess.run([sys.executable, "-c", _CAPTURE, ROOT, start], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
