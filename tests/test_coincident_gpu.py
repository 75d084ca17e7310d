"""Members at exactly the same FP32 position (snapshots stored in single
precision): the spline-softened kernel is finite at distance 0, on plain and
refined particle-mesh halos and both precisions.  First-pass potentials
against the CPU oracle (tolerance as in test_pm_gpu.py: 1e-5 of the halo's
largest |phi|), and a whole call."""
import numpy as np
import pytest

import py_fof_b200 as P
from oracle import oracle as O
from py_fof_b200 import _native
from tests.helpers import check_unbinding_band, oracle_core_diag
from tests.test_pm_gpu import S15, _pm_halos
from tests.test_short_range_gpu import _ball

pytestmark = pytest.mark.gpu


def _cases():
    x = _ball(1300, 0.4, 1)
    x[:, 700] = x[:, 20]
    yield "one_pair", x
    x = _ball(2400, 0.3, 2)
    x[:, 1200:] = x[:, :1200]  # every position twice
    yield "all_twice", x
    x = np.concatenate([_ball(16000, 0.35, 3, (0.1, 0.2, -0.3)), np.random.default_rng(4).uniform(-5, 5, (3, 800))],
                       axis=1)
    x[:, 8000:9000] = x[:, :1000]
    yield "refined", x


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("name,x", list(_cases()), ids=[c[0] for c in _cases()])
def test_first_pass_potential(name, x, fp64):
    n = x.shape[1]
    q = (x - x[:, :1]).astype(np.float32)
    w = np.random.default_rng(n).lognormal(-0.045, 0.3, n).astype(np.float32)
    xv = np.zeros((n, 6), np.float32)
    xv[:, :3] = q.T
    g_o, phi_o = O.first_potential(xv, w, np.arange(1, n + 1), softening=0.1, a_val=1.0, s15=S15)
    phi, g = _native.halo_potential(q, w, fp64=fp64, s15=S15)
    assert g == g_o > 0
    if name == "refined":
        assert _native.get_stat("refined_regions") > 0
    assert np.abs(phi - phi_o).max() < 1e-5 * np.abs(phi_o).max()


@pytest.mark.parametrize("fp64", [1, 0])
def test_unbinding(fp64):
    xs, vs, ms = _pm_halos(41, [1500, 3000])
    for x in xs:
        x[:, 400:500] = x[:, :100]
    kw = dict(vp_list=vs, mp_list=ms, L_Box=512.0, linking_length=0.3, np_halo_min=10, bound_check=True)
    o, energy, scale = oracle_core_diag(xs, **kw)
    with _native.options(unbind_fp64=fp64):
        check_unbinding_band(P._fof_core(xs, **kw), o, energy, scale)
