"""Large pageable positions with velocities or masses in device memory (the
runtime's copy takes either): the copy threads read host memory only, so such
a call must not reach them.  In a process of its own, since it crashed."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import ctypes
import numpy as np
import torch
from py_fof_b200 import _native
n = 700000
rng = np.random.default_rng(1)
x = rng.uniform(0, 20.0, (3, n))
v = rng.normal(0, 1.0, (3, n))
m = rng.uniform(0.5, 2.0, n)
dv, dm = torch.from_numpy(v).cuda(), torch.from_numpy(m).cuda()
nph = np.array([n], np.int32)
L = _native.load()
D, I = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int32)

def run(vp, mp):
    ids, am = np.full(n, 7, np.int32), np.zeros((3, 1), order="F")
    r = L.pyfof_run(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(vp), ctypes.c_void_p(mp), 0,
                    nph.ctypes.data_as(I), 1, n, 20.0, 0.15, 5, 0, 0, 0.1, 1.0, 0.0, 17.0, 0, 256, 512.0, None,
                    ctypes.c_void_p(ids.ctypes.data), am.ctypes.data_as(D))
    assert r == 0, _native.last_error()
    return ids, am

want = run(v.ctypes.data, m.ctypes.data)
assert want[0].max() > 100
for vp, mp in ((dv.data_ptr(), m.ctypes.data), (v.ctypes.data, dm.data_ptr()), (dv.data_ptr(), dm.data_ptr())):
    got = run(vp, mp)
    assert np.array_equal(got[0], want[0])
    assert np.allclose(got[1], want[1], rtol=1e-9, atol=1e-9 * np.abs(want[1]).max())
print("same")
"""


def test_device_velocities_and_masses():
    p = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, (p.returncode, p.stderr)
    assert p.stdout == "same\n", p.stdout
