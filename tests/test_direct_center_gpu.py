"""The direct-summation path at the sizes of its target groups and blocks, and
where its parallel centre sums cannot settle the FP32 centre (members mirrored
about the centre, so that the sums cancel) and the ordered sums run instead.
The FP64 path equals the oracle bit for bit."""
import numpy as np
import pytest

import py_fof_b200 as P
from py_fof_b200 import _native
from tests.helpers import check_unbinding_band, oracle_core_diag

pytestmark = pytest.mark.gpu

SIZES = [10, 11, 31, 32, 33, 63, 64, 65, 127, 129, 255, 257, 449, 511, 513, 999, 1000]


def _halos(mirror):
    rng = np.random.default_rng(17 + mirror)
    xs, vs, ms = [], [], []
    for n in SIZES:
        d = rng.standard_normal((3, n)) * 0.25
        v = rng.standard_normal((3, n)) * np.sqrt(0.02 * n)
        m = rng.lognormal(0.0, 0.3, n)
        d[:, 0] = v[:, 0] = 0.0
        if mirror:
            h = (n - 1) // 2
            d[:, 1:1 + h], v[:, 1:1 + h] = -d[:, n - h:], -v[:, n - h:]
            m[1:1 + h] = m[n - h:]
            if n % 2 == 0:
                d[:, 1 + h], v[:, 1 + h] = 0.01, 0.0
        xs.append(d + rng.uniform(50, 450, (3, 1)))
        vs.append(v)
        ms.append(m)
    return xs, vs, ms


@pytest.mark.parametrize("mirror", [False, True])
def test_direct_matches_oracle(mirror):
    xs, vs, ms = _halos(mirror)
    kw = dict(vp_list=vs, mp_list=ms, L_Box=512.0, linking_length=0.5, np_halo_min=5, bound_check=True,
              return_ang_mom=True)
    o, energy, scale = oracle_core_diag(xs, **kw)
    assert 0.1 < o[0].mean() < 0.999 and int(o[1].max()) > 10
    g = P._fof_core(xs, **kw)
    assert _native.get_stat("direct_halos") >= len(SIZES)
    assert np.array_equal(g[0], o[0]) and np.array_equal(g[1], o[1])
    with _native.options(unbind_fp64=0):
        check_unbinding_band(P._fof_core(xs, **kw), o, energy, scale)


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 33, 255, 256, 257, 1000])
def test_first_pass_is_the_static_path(n):
    """halo_potential (targets shared by lanes) against the one-block kernel
    of the allocation-free entry point: the same bits."""
    rng = np.random.default_rng(n)
    q = rng.standard_normal((3, n)).astype(np.float32)
    q -= q[:, :1]
    w = rng.lognormal(0.0, 0.3, n).astype(np.float32)
    for fp64 in (True, False):
        a, meth = _native.halo_potential(q, w, fp64=fp64)
        b, ierr = _native.halo_potential_direct_static(q, w, fp64=fp64)
        assert meth == 0 and ierr == 0
        assert np.array_equal(a, b)


@pytest.mark.parametrize("fp64", [1, 0])
def test_first_pass_of_many_halos_is_that_of_few(fp64):
    """More direct-summation members in a call than the chip has thread slots
    (a lane per target) against the same halos in two calls that stay below
    (eight lanes per target in FP64): the same bits."""
    rng = np.random.default_rng(5)
    sizes = rng.integers(700, 1000, 480)
    xs = [rng.standard_normal((3, n)) * 0.25 + rng.uniform(50, 450, (3, 1)) for n in sizes]
    vs = [rng.standard_normal((3, n)) * np.sqrt(0.02 * n) for n in sizes]
    kw = dict(L_Box=512.0, linking_length=0.5, np_halo_min=5, bound_check=True)
    h = len(sizes) // 2
    assert sizes.sum() > 148 * 2048 > max(sizes[:h].sum(), sizes[h:].sum())
    with _native.options(unbind_fp64=fp64):
        g = P._fof_core(xs, vp_list=vs, **kw)
        assert _native.get_stat("direct_halos") >= len(sizes)
        parts = [P._fof_core(xs[a:b], vp_list=vs[a:b], **kw) for a, b in ((0, h), (h, len(sizes)))]
    in_halo, halo_id = np.asarray(g[0]), np.asarray(g[1])
    assert 0.1 < in_halo.mean() < 0.999
    assert np.array_equal(in_halo, np.concatenate([q[0] for q in parts]))
    assert np.array_equal(halo_id > 0, np.concatenate([q[1] for q in parts]) > 0)
