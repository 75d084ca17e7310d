"""An error that a direct-summation halo reports while the tables of the
particle-mesh halos are being built (the first call of a process) must end the
call: the tables have a status word of their own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import numpy as np
from py_fof_b200 import _native
rng = np.random.default_rng(1)
x = np.concatenate([20.0 + 0.05 * rng.standard_normal((3, 30)), 60.0 + 0.4 * rng.standard_normal((3, {n}))], axis=1)
v = np.zeros_like(x)
v[0, 0] = 1e25  # its energy overflows FP32
n = x.shape[1]
r = _native.run(x, v, None, np.array([n], np.int32), 1, 100.0, 0.3, 10, 1, 0, 0.1, 1.0, 0.0, 17.0, 0, n)
assert _native.get_stat("direct_halos") == 1 and _native.get_stat("pm_halos") == 1
print("ierr", r[3], _native.last_error())
v[0, 0] = 0.0
r = _native.run(x, v, None, np.array([n], np.int32), 1, 100.0, 0.3, 10, 1, 0, 0.1, 1.0, 0.0, 17.0, 0, n)
print("then", r[3], int(r[1].max()))
"""


@pytest.mark.parametrize("n", [1500, 30000])  # 30,000: with refined regions, whose tables come later
def test_error_survives_the_table_build(n):
    p = subprocess.run([sys.executable, "-c", CODE.format(n=n)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    lines = p.stdout.splitlines()
    assert lines[0].startswith("ierr ") and int(lines[0].split()[1]) != 0, p.stdout
    assert "Green" not in lines[0], p.stdout
    assert lines[1] == "then 0 2", p.stdout
