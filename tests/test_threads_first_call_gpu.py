"""Several threads whose first few-row call comes at the same moment: what the library finds out about the device on that occasion must not
change how a call splits its sum, so all threads get the same bits.  A process of its own, because the answer is kept."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = r"""
import sys, threading
import torch
from zendnn_b200 import capi
M, K, N, T = 8, 8192, 2048, 8
w, x = (torch.randn(K, N, device="cuda") * 0.02).bfloat16(), torch.randn(M, K, device="cuda").bfloat16()
outs, streams = [torch.zeros(M, N, device="cuda") for _ in range(T)], [torch.cuda.Stream() for _ in range(T)]
kw = dict(src_dt=capi.DT["bf16"], wei_dt=capi.DT["bf16"], dst_dt=capi.DT["f32"])
big = torch.randn(200, K, device="cuda").bfloat16()
warm = torch.zeros(200, N, device="cuda")
d = capi.make_matmul(200, N, K, big, w, warm, **kw)       # the tile kernel: weight packed, every stream's context made
for s in streams:
    capi.check(capi.matmul(d, s.cuda_stream))
    torch.cuda.synchronize()
descs = [capi.make_matmul(M, N, K, x, w, o, **kw) for o in outs]
gate = threading.Barrier(T)
def run(i):
    gate.wait()
    capi.check(capi.matmul(descs[i], streams[i].cuda_stream))
threads = [threading.Thread(target=run, args=(i,)) for i in range(T)]
[t.start() for t in threads]; [t.join() for t in threads]
torch.cuda.synchronize()
sys.exit(0 if all(torch.equal(outs[0], o) for o in outs) else 3)
"""


def test_first_calls_of_several_threads_agree():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", CODE], cwd=root, capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stderr[-2000:] or "the threads' results differ"
