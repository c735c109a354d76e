"""Threads that create the process's first contexts at the same time: each
returns with its kernels' shared-memory limits raised, so each can launch.  A
child process per round, since only a process's first creation raises them."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
CHILD = r"""
import sys, threading
import numpy as np
import torch
import cbns3d_cuda_b200 as cb

torch.zeros(1, device="cuda")  # the GPU's context, but none of the library's
precision, n = int(sys.argv[1]), 8
k, j, i = np.meshgrid(*(np.linspace(0.0, 1.0, 8),) * 3, indexing="ij")
Q = np.ones((12, 12, 12, 5))
Q[..., 1:4], Q[..., 4] = 0.1, 2.5
start, errors = threading.Barrier(n), []

def work():
    try:
        p = cb.make_params(8, 8, 8, precision=precision, bc_mode=cb.BC_FARFIELD)
        start.wait()
        b = cb.Block(p)
        b.calc_metrics(i, j, k)
        b.set_conservative(Q)
        b.eval_rhs()
    except Exception as e:
        errors.append(str(e))

ts = [threading.Thread(target=work) for _ in range(n)]
for t in ts: t.start()
for t in ts: t.join()
print("\n".join(errors))
sys.exit(1 if errors else 0)
"""


@pytest.mark.parametrize("precision", [0, 1])
def test_first_contexts_from_several_threads(precision):
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", CHILD, str(precision)], cwd=ROOT, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
