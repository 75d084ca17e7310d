"""Pageable inputs large enough to be copied by worker threads: the same
results as the same inputs in page-locked memory (copied directly), in both
layouts, with masses, velocities and unit conversion, from concurrent slots,
and when the call fails before it needs the later inputs."""
import threading

import numpy as np
import pytest

import py_fof_b200 as P
from py_fof_b200 import _native, workloads as W

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch
    t = torch.empty(a.shape if a.flags.c_contiguous else a.T.shape, dtype=torch.float64, pin_memory=True)
    b = t.numpy()
    b[...] = a if a.flags.c_contiguous else a.T
    return (b if a.flags.c_contiguous else b.T), t


def _box(n_side=84):
    return W.plummer_box(n_side ** 3 + 77, float(n_side), 40, seed=2, with_velocities=True, lognormal_mass=0.3)


@pytest.mark.parametrize("aos", [False, True])
@pytest.mark.parametrize("bound", [False, True])
def test_pageable_equals_pinned(aos, bound):
    d = _box()
    x, v, m = d["xp"], d["vp"], d["mp"]
    if aos:
        x, v = np.asfortranarray(x), np.asfortranarray(v)
    kw = dict(linking_length=0.2, np_halo_min=20, bound_check=bound, softening=0.1, ng_global=256.0,
              return_ang_mom=True, L_Box=84.1)
    a = P._fof_core(x, v, mp_list=m, **kw)
    (px, k1), (pv, k2), (pm, k3) = _pinned(x), _pinned(v), _pinned(m)
    b = P._fof_core(px, pv, mp_list=pm, **kw)
    assert a[0].sum() > 1000
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    assert np.allclose(a[2], b[2], rtol=1e-9, atol=1e-9 * np.abs(b[2]).max())


def test_units_and_constant_mass():
    d = _box()
    dx = 300.0 / 512.0
    kw = dict(units="physical", L_Box=300.0, n_sim=512 ** 3, linking_length=0.2 * dx, softening=0.1 * dx,
              bound_check=True, return_ang_mom=True)
    x, v = d["xp"] * dx, d["vp"] * 10.0
    a = P.fof(x, v, **kw)
    (px, k1), (pv, k2) = _pinned(x), _pinned(v)
    b = P.fof(px, pv, **kw)
    assert np.array_equal(a[0], b[0])
    assert np.allclose(a[1], b[1], rtol=1e-9, atol=1e-9 * np.abs(b[1]).max())


def test_slots_and_errors():
    d = _box()
    n = d["xp"].shape[1]
    args = lambda x: (x, d["vp"], d["mp"], np.array([n], np.int32), 1, 84.1, 0.2, 20, 1, 0, 0.1, 1.0, 0.0, 8.5, 0, n)  # noqa: E731
    want = _native.run(*args(d["xp"]))
    assert want[3] == 0
    bad = d["xp"].copy()
    bad[1, 5] = np.nan  # fails before masses and velocities are waited for
    slots = [_native.slot_create() for _ in range(3)]
    got = [None] * 3
    try:
        def job(i):
            for _ in range(2):
                assert _native.run(*args(bad), slot=slots[i])[3] == 4
                got[i] = _native.run(*args(d["xp"]), slot=slots[i])
        th = [threading.Thread(target=job, args=(i,)) for i in range(3)]
        for t in th:
            t.start()
        for t in th:
            t.join()
    finally:
        for s in slots:
            _native.slot_destroy(s)
    for g in got:
        assert g is not None and g[3] == 0
        assert np.array_equal(g[1], want[1])
