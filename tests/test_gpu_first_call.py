"""Kernels that are loaded when they are first needed, in a process of their own: the first call, and the first call captured."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys, torch
from nebula_b200 import api
h = api.Handle(0, "fp32")
g = torch.Generator(device="cuda").manual_seed(0)
a, b = torch.randn(70, 96, device="cuda", generator=g), torch.randn(80, 96, device="cuda", generator=g)
c = torch.zeros(70, 80, device="cuda")
fc = api.Connected(h, 70, 96, 80, False, "linear")
fc.set_weights(b, torch.zeros(80, device="cuda"))
fc.prepare()
out = torch.zeros(70, 80, device="cuda")
def calls():
    h.gemm(False, True, 70, 80, 96, 1.0, a, 96, b, 96, 0.0, c, 80)
    h.check(h.lib.nb_fc_forward(fc.p, a.data_ptr(), out.data_ptr()))
torch.cuda.synchronize()
if sys.argv[1] == "captured":
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        calls()
    h.set_stream(0)
    graph.replay()
else:
    calls()
torch.cuda.synchronize()
h.synchronize()
ref = a.double() @ b.double().T
for y in (c, out):
    assert float((y - ref).abs().max() / ref.abs().max()) < 1e-5
print("OK")
"""


@pytest.mark.parametrize("how", ["launched", "captured"])
def test_first_call_of_a_process(how):
    env = dict(os.environ, PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", CHILD, how], capture_output=True, text=True, timeout=300, env=env, cwd=ROOT)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stderr[-2000:]
