"""Convolutions over each halo's own support box: halos stretched along one
axis, flat ones, ones that fill their grid to the last node and a mix in one
call, on every grid size.  First-pass potentials against the CPU oracle,
which transforms the whole grid (tolerance as in test_pm_gpu.py: 1e-5 of the
halo's largest |phi|)."""
import numpy as np
import pytest

import py_fof_b200 as P
from oracle import oracle as O
from py_fof_b200 import _native
from tests.helpers import check_unbinding_band, oracle_core_diag

pytestmark = pytest.mark.gpu

S15 = 15 * 0.67 * 512 / 300.0
# (members, extent) whose reference grid is 48, 64, 128 and 256 (spacing
# 0.125 / 0.125 / 0.25 / 0.0625 covers just above the extent)
GRIDS = [(1200, 2.6), (1300, 3.6), (1100, 15.2), (6000, 7.8)]


@pytest.mark.parametrize("n,extent", GRIDS)
@pytest.mark.parametrize("shape", [(1.0, 0.1, 0.02), (0.02, 1.0, 0.3), (0.2, 0.05, 1.0), (0.01, 1.0, 1.0),
                                   (1.0, 1.0, 1.0)])
def test_potential_of_shapes(n, extent, shape):
    rng = np.random.default_rng(n)
    x = rng.random((3, n)) * np.array(shape)[:, None] * extent
    x[:, 1] = 0.0  # both corners of the box are occupied
    x[:, 2] = np.array(shape) * extent * (1 - 1e-6)
    q = (x - x[:, :1]).astype(np.float32)
    w = rng.lognormal(-0.045, 0.3, n).astype(np.float32)
    xv = np.zeros((n, 6), np.float32)
    xv[:, :3] = q.T
    g_o, phi_o = O.first_potential(xv, w, np.arange(1, n + 1), softening=0.1, a_val=1.0, s15=S15)
    scale = np.abs(phi_o).max()
    for fp64 in (True, False):
        phi, g = _native.halo_potential(q, w, fp64=fp64, s15=S15)
        assert g == g_o > 0
        err = np.abs(phi - phi_o).max() / scale
        assert err < 1e-5, (fp64, err)


def test_mixed_batch():
    """Halos of different shapes and sizes batched on the same grids."""
    rng = np.random.default_rng(8)
    xs, vs = [], []
    for k, n in enumerate([1100, 1300, 1250, 2200, 4100, 6000]):
        s = np.array([1.0, 0.2 + 0.15 * k, 1.0 - 0.13 * k])
        xs.append(rng.random((3, n)) * s[:, None] * 1.6 + rng.uniform(50, 450, (3, 1)))
        vs.append(rng.standard_normal((3, n)) * 4.0)
    kw = dict(vp_list=vs, L_Box=512.0, linking_length=0.4, np_halo_min=10, bound_check=True, return_ang_mom=True)
    g = P._fof_core(xs, **kw)
    assert _native.get_stat("pm_halos") >= 5
    o, energy, scale = oracle_core_diag(xs, **kw)
    check_unbinding_band(g, o, energy, scale)
