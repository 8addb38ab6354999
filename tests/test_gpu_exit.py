"""A program that ends with a batch and its operators alive ends cleanly: what belongs to
a context is freed before it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r'''
import sys
sys.path[:0] = [{root!r}, {root!r} + "/quantumopticsbase.jl_gb300"]
import torch
import qobgpu as Q
from qobgpu.evolution import Batch
from qobgpu.hamiltonians import two_mode_cavity
batch = Batch()
keep = []
for k in range(4):
    H = two_mode_cavity(5 + k, 6, seed=k)
    x = torch.ones(len(H.basis_l), dtype=torch.complex128, device="cuda:0")
    y = torch.zeros_like(x)
    batch.add(H, x, y, 1.0, 0.0)
    keep.append((H, x, y))
batch.run()
torch.cuda.synchronize()
assert all(float(y.abs().sum()) > 0 for _, _, y in keep)
gone = Batch()
gone.add(*keep[0], 1.0, 0.0)
gone.run()
del gone
print("ok")
'''


def test_exit_with_a_batch_alive():
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout[-500:], r.stderr[-2000:])
