"""Tensor-core kernels that are loaded when a plan or a launch first needs them, in a process of their own: plain epilogues, folded
shortcuts, gathered inputs, clusters, slabs and the recurrences, called and captured."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys, torch
import numpy as np
from nebula_b200 import api
from nebula_b200.workloads import NetBuilder
how, mode = sys.argv[1], sys.argv[2]
h = api.Handle(0, mode)
g = torch.Generator(device="cuda").manual_seed(0)
def N(*s): return torch.randn(*s, device="cuda", generator=g)
plans, ins, outs, f = [], [], [], []
def add(plan, x, n, fwd):
    y = torch.full((n,), 7.0, device="cuda")
    plan.prepare()
    plans.append(plan); ins.append(x); outs.append(y)
    f.append(lambda: h.check(fwd(plan.p, x.data_ptr(), y.data_ptr())))
for B, C, S, F, k in ((2, 64, 40, 64, 3), (2, 6, 30, 40, 5), (1, 256, 14, 256, 3), (4, 3, 33, 64, 3)):
    p = api.Conv2d(h, B, C, S, S, F, k, 1, k // 2, False, "relu")
    p.set_weights(N(F, C, k, k) / (C * k * k) ** 0.5, N(F))
    add(p, N(B, C, S, S), B * F * S * S, h.lib.nb_conv2d_forward)
for B, i, o in ((70, 96, 80), (5, 1200, 60), (4, 40000, 32)):
    p = api.Connected(h, B, i, o, False, "linear")
    p.set_weights(N(o, i) / i ** 0.5, N(o))
    add(p, N(B, i), B * o, h.lib.nb_fc_forward)
def calls():
    for c in f: c()
torch.cuda.synchronize()
if how == "captured":
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
first = [y.clone() for y in outs]
calls()
h.synchronize()
assert all(torch.equal(a, b) and bool((a != 7.0).any()) and bool(a.isfinite().all()) for a, b in zip(first, outs))
# a folded shortcut of many tiles, through the executor
b = NetBuilder("n", 8, channels=64, height=56, width=56, bias_init="bias_n01")
b.conv(64, 1, 1, 0, "relu"); b.conv(256, 1, 1, 0, "linear"); b.conv(64, 1, 1, 0, "relu"); b.conv(256, 1, 1, 0, "linear"); b.shortcut(3, "relu"); b.connected(10, "linear")
wl = b.build("normal")
net = api.Network(h, wl.cfg)
net.load_weights(wl.make_weights(1))
x = torch.from_numpy(wl.make_input(2)).cuda()
if how == "captured": net.set_graph(True)
net.forward(x); a = net.logits("cuda").clone()
net.forward(x)
assert torch.equal(a, net.logits("cuda")) and bool(a.isfinite().all())
h.synchronize()
print("OK")
"""


@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("how", ["launched", "captured"])
def test_first_call_of_a_process(how, mode):
    env = dict(os.environ, PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", CHILD, how, mode], capture_output=True, text=True, timeout=300, env=env, cwd=ROOT)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stderr[-2000:]
