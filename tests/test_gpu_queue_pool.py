"""Device memory that the batched launches' work queue keeps is given back.

In a process of its own: the last handle to go gives it back, and other tests'
handles may still live here.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import torch
import entropydecreaseboltzmann_gb300 as edb

N, S = 8, 4096
fin = torch.randn(S, N ** 3, dtype=torch.complex64, device="cuda")
out = torch.empty_like(fin)

def run(solves):
    q = edb.QCalculator(N, 0, gamma=0.0, L=6.0, filter=False, index_mode=edb.INDEX_ALIASED)
    q.genB()
    for _ in range(2):
        q.calQ_batch_f32_ex(solves, 0, 1, None, fin, out)
    torch.cuda.synchronize()
    del q
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

run(16)           # loads the kernels; a grid that holds every item has no queue
free = run(16)
assert run(S) >= free, (free, run(S))
"""


def test_the_last_handle_gives_the_pool_back():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
