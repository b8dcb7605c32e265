"""The first call of a process under stream capture: what a call sets up on first use has to be allowed there."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MATMUL = """
import torch
from lapis_b200 import device
m, n, k = {shape}
A, B, C = (torch.randint(-4, 5, s, device="cuda").float() for s in ((m, k), (k, n), (m, n)))
out = C.clone()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    device.bgemm(A, B, out)
assert torch.equal(out, C)
want = (C.double() + A.double() @ B.double()).float()
for _ in range(2):
    out.copy_(C)
    graph.replay()
    assert torch.equal(out, want)
device.bgemm_status()
out.copy_(C)
assert torch.equal(device.bgemm(A, B, out), want)
print("done")
"""


@pytest.mark.parametrize("shape", [(40, 50, 60), (1000, 1501, 777), (2100, 2099, 8000), (128, 128, 32), (1024, 1536, 2048)])
def test_matmul(shape):
    """The kernel for general shapes, both products from split operands, one of several groups, and the kernel for whole tiles."""
    r = subprocess.run([sys.executable, "-c", MATMUL.format(shape=shape)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "done\n", r.stdout + r.stderr[-2000:]
