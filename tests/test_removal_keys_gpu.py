"""The key buffer of the one-block removal loop (4096 keys) with a known
number of unbound members in the first sweep: cold members are bound whatever
their place, hot ones unbound, so the hot ones' number is the sweep's."""
import numpy as np
import pytest

import py_fof_b200 as P
from py_fof_b200 import _native
from tests.helpers import check_unbinding_band, oracle_core_diag
from tests.test_pm_gpu import plummer

pytestmark = pytest.mark.gpu

N = 12000


@pytest.mark.parametrize("hot", [4095, 4096, 4097, 7000])
def test_first_sweep_at_the_buffer(hot):
    rng = np.random.default_rng(hot)
    x, _ = plummer(N, 1.0, 77, rmax=4.0)
    phi, _ = _native.halo_potential((x - x[:, :1]).astype(np.float32), np.ones(N, np.float32), fp64=True)
    depth = np.sqrt(2.0 * np.abs(phi))  # escape speeds
    v = np.zeros((3, N))
    k = rng.permutation(N)[:hot]
    d = rng.standard_normal((3, hot))
    d /= np.linalg.norm(d, axis=0)
    v[:, k] = d * depth.max() * rng.uniform(3.0, 6.0, hot)
    vc = v.mean(axis=1, keepdims=True)
    energy = 0.5 * ((v - vc) ** 2).sum(axis=0) + phi
    assert (energy >= 0).sum() == hot and np.abs(energy / np.abs(phi)).min() > 0.5
    kw = dict(vp_list=v, L_Box=512.0, linking_length=0.5, np_halo_min=10, bound_check=True)
    o, en, scale = oracle_core_diag(x + 256.0, **kw)
    for fp64 in (1, 0):
        with _native.options(unbind_fp64=fp64):
            check_unbinding_band(P._fof_core(x + 256.0, **kw), o, en, scale)
            assert _native.get_stat("candidates") == 1 and _native.get_stat("active") == N
