"""First calls of a process from several threads at once, in a child process."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_CHILD = """
import threading, torch
from t81lib_b200 import ops
trits = torch.randint(-1, 2, (300, 400), device="cuda").float()
t2 = ops.pack_t2(ops.quantize_pack(trits, 0.5, "fixed")[0], 300, 400)
x = torch.randint(-3, 4, (64, 400), device="cuda").to(torch.bfloat16)
want = x.float() @ trits.t()
torch.cuda.synchronize()
start, good = threading.Barrier(16), []
def call():
    start.wait()
    y = ops.linear_t2(t2, 300, x, 400, None, None, torch.float32)  # the process's first tensor map
    torch.cuda.synchronize()
    good.append(torch.equal(y, want))
threads = [threading.Thread(target=call) for _ in range(16)]
[t.start() for t in threads]
[t.join() for t in threads]
assert good == [True] * 16, good
print("worker ok")
"""


def test_first_tensor_maps_of_many_threads(lib_built):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", _CHILD], capture_output=True, text=True, timeout=300, cwd=root)
    assert res.returncode == 0 and "worker ok" in res.stdout, res.stdout + res.stderr
