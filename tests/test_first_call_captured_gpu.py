"""The first library call of a process may be one that a stream capture records: the
Sobel filter on a layout that TMA cannot address, and a local operator on 16-bit
storage, which take the device's status word and counters but no scratch.  Each runs
in a process of its own; the replayed graph gives what the call gives uncaptured."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CALLS = {
    "sobel": """
x = torch.randint(0, 256, (75, 101), dtype=torch.uint8, device="cuda")
call = lambda y: api.sobel_mag(x, y)
""",
    "conv_bf16": """
x = torch.rand((64, 128), device="cuda").to(torch.bfloat16)
call = lambda y: api.local_op(x, y, mask=np.full((5, 5), 0.04, np.float32))
""",
}
PROGRAM = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
import torch
from hipacc_gb300 import api
torch.manual_seed(0)
{call}
captured, plain = torch.zeros_like(x), torch.zeros_like(x)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    call(captured)
graph.replay()
call(plain)
torch.cuda.synchronize()
assert plain.any() and torch.equal(captured, plain)
"""


@pytest.mark.parametrize("name", sorted(CALLS))
def test_first_call_of_a_process_is_captured(hgb_lib, name):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT, call=CALLS[name])], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
