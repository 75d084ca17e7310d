"""The removal loops of the particle-mesh halos where their parts change:
halos of a few blocks of members, unbound members below and above the
one-block loop's key buffer (4096), and the chunked loop on the same halos,
against the oracle."""
import numpy as np
import pytest

import py_fof_b200 as P
from py_fof_b200 import _native
from tests.helpers import check_unbinding_band, oracle_core_diag
from tests.test_pm_gpu import _pm_halos

pytestmark = pytest.mark.gpu

KEYS = 4096


@pytest.mark.parametrize("n,hot,over", [(6000, 0.3, False), (16000, 0.2, True), (16000, 0.5, True)])
def test_removal_loops_match_oracle(n, hot, over):
    xs, vs, ms = _pm_halos(31, [1500, 2100, 4200, n])
    rng = np.random.default_rng(n)
    k = rng.choice(n, int(hot * n), replace=False)
    vs[-1][:, k] *= 6.0
    kw = dict(vp_list=vs, mp_list=ms, L_Box=512.0, linking_length=0.3, np_halo_min=10, bound_check=True)
    o, energy, scale = oracle_core_diag(xs, **kw)
    left = n - int(o[0][-n:].sum())
    assert (left > KEYS) == over, left
    with _native.options(unbind_fp64=1):
        a = P._fof_core(xs, **kw)
        assert _native.get_stat("pm_halos") >= 3
        with _native.options(unbind_big_np=1000):
            b = P._fof_core(xs, **kw)
    check_unbinding_band(a, o, energy, scale)
    check_unbinding_band(b, o, energy, scale)
    with _native.options(unbind_fp64=0):
        check_unbinding_band(P._fof_core(xs, **kw), o, energy, scale)
