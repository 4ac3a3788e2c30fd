"""Memory that a one-shot batch leaves behind, on the GPU."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# In a process of its own, so that no earlier call has grown the kept buffers: a small
# batch, then n boards that are all distinct and have no free column (no subtask, but
# two result words each), and the device memory that the second call kept.
SCRIPT = """
import ctypes, sys
import numpy as np, torch
sys.path.insert(0, {root!r})
import n_queens_b200 as nq
n = {n}
nq.count_batch([(12, 0, 0, 0)])
b = np.zeros((n, 4), np.uint32)
b[:, 0] = 24
b[:, 1] = np.arange(n) + 1
b[:, 2] = (1 << 24) - 1
inst = (nq.Instance * n).from_buffer(b)
out = np.full(n, 7, np.uint64)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
assert nq.lib.nq_count_batch(inst, n, 0, nq._p(out, nq._u64p), None, None) == 0
assert not out.any()
print(free - torch.cuda.mem_get_info()[0])
"""


# 2^20 and 2^21 boards: 16 and 32 MiB of result words.
@pytest.mark.parametrize("n", [(1 << 20) + 1, 1 << 21])
def test_one_shot_batch_of_dead_boards_gives_its_memory_back(gpu, n):
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT, n=n)], capture_output=True, text=True,
                       timeout=300, cwd=os.path.dirname(ROOT))
    assert r.returncode == 0, r.stderr
    assert int(r.stdout.split()[-1]) <= 4 << 20
