"""The kernel tables at shorter transform lengths are an extra: a device with
too little free memory for them (another framework holds it) still unbinds
256-grid halos, at the full length.  In a process of its own, with all but 460
MB of the device taken: the 256-point table and the transform that makes it
need 345 MB, the shorter tables 166 MB while they are made."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import numpy as np
import torch
from oracle import oracle as O
from py_fof_b200 import _native
S15 = 15 * 0.67 * 512 / 300.0
rng = np.random.default_rng(1)
_native.halo_potential(rng.normal(0, 0.1, (3, 50)), np.ones(50), fp64=True, s15=S15)  # the context's own memory
free, _ = torch.cuda.mem_get_info()
held = torch.empty(free - (460 << 20), dtype=torch.uint8, device="cuda")
n = 21000
x = np.clip(rng.normal(0, 0.8, (3, n)), -2.5, 2.5)
q = (x - x[:, :1]).astype(np.float32)
w = np.ones(n, np.float32)
xv = np.zeros((n, 6), np.float32)
xv[:, :3] = q.T
g_o, want = O.first_potential(xv, w, np.arange(1, n + 1), softening=0.1, a_val=1.0, s15=S15)
phi, g = _native.halo_potential(q, w, fp64=True, s15=S15)
assert g == g_o == 4, (g, g_o)
err = np.abs(phi - want).max() / np.abs(want).max()
assert err < 1e-5, err
print("bound", torch.cuda.mem_get_info()[0] >> 20)
"""


def test_without_room_for_the_shorter_tables():
    p = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    assert p.stdout.startswith("bound "), p.stdout
