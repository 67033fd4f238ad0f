"""The first forward pass of a process: what it loads, and that a stream capture may be that pass."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import time, torch
from n2d2_b200 import netdesc, runtime
net = netdesc.resnet50(size=64, classes=100)
qn = runtime.QuantizedNet(net, 3)
x = torch.from_numpy(netdesc.make_input(net, 3)).cuda()
y = torch.zeros((3, qn.out_elems), dtype=torch.uint8, device='cuda')
torch.cuda.synchronize()
"""


def _fresh_process(code):
    run = subprocess.run([sys.executable, '-c', PRELUDE + code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    return run.stdout.split()


def test_first_call_loads_only_the_kernels_it_launches():
    # kernel code lives in device memory from its first use on: the variants of a ResNet's pass take about 2 MiB, the whole tables of
    # variants that they are picked from three times that
    out = _fresh_process("""
free = torch.cuda.mem_get_info()[0]
qn.forward_device(x.data_ptr(), 3, y.data_ptr())
torch.cuda.synchronize()
print(free - torch.cuda.mem_get_info()[0])
""")
    assert int(out[0]) <= 4 << 20


def test_first_call_may_be_a_stream_capture():
    out = _fresh_process("""
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    qn.forward_device(x.data_ptr(), 3, y.data_ptr(), torch.cuda.current_stream().cuda_stream)
graph.replay()
torch.cuda.synchronize()
captured = y.clone()
y.zero_()
qn.forward_device(x.data_ptr(), 3, y.data_ptr())
qn.check()
print(bool((captured == y).all()), bool(captured.any()))
""")
    assert out == ['True', 'True']
