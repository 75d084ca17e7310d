"""Particles in arbitrary order inside their cell: the halo numbering and
first members must still be the reference's.  Several groups rooted in one
cell, coordinates exactly on cell boundaries and box edges, coordinates
periods away, list inputs with skipped regions.  Equal to the oracle, on
every repetition."""
import numpy as np
import pytest

import py_fof_b200 as P
from tests.helpers import oracle_core

pytestmark = pytest.mark.gpu


def _check(x, rep=3, **kw):
    o = oracle_core(x, **kw)
    assert o[1].max() > 1
    for _ in range(rep):
        g = P._fof_core(x, **kw)
        assert np.array_equal(g[0], o[0]) and np.array_equal(g[1], o[1])


@pytest.mark.parametrize("np_min", [1, 2, 10])
@pytest.mark.parametrize("n_groups", [300, 3000])
def test_groups_sharing_a_cell(np_min, n_groups):
    # cells are about three links wide (set by the mean density), groups a
    # tenth of a link: many groups per cell, members interleaved in index
    rng = np.random.default_rng(n_groups + np_min)
    L = 12.0
    cen = rng.uniform(0, L, (3, n_groups))
    x = np.repeat(cen, 12, axis=1) + rng.normal(0, 0.004, (3, 12 * n_groups))
    x = np.mod(x[:, rng.permutation(x.shape[1])], L)
    _check(x, L_Box=L, linking_length=0.05, np_halo_min=np_min)


@pytest.mark.parametrize("side", [4, 10, 16])
def test_lattice_on_cell_boundaries(side):
    # a lattice commensurate with the cells, jittered pairs on its points
    rng = np.random.default_rng(side)
    g = np.stack(np.meshgrid(*[np.arange(side, dtype=np.float64)] * 3, indexing="ij"), 0).reshape(3, -1)
    x = np.concatenate([g, g + np.array([0.0, 0.125, 0.0])[:, None], g[:, ::3] + 0.1], axis=1)
    x = x[:, rng.permutation(x.shape[1])]
    _check(np.mod(x, side), L_Box=float(side), linking_length=0.2, np_halo_min=2)
    _check(x + 37.0, L_Box=1000.0, linking_length=0.2, np_halo_min=2)


def test_coordinates_periods_away():
    rng = np.random.default_rng(3)
    x = rng.uniform(0, 10.0, (3, 4000))
    x[:, ::5] += 10.0 * rng.integers(-4, 5, (3, 800))
    x[:, :3] = np.array([[0.0, 10.0, -10.0], [5.0, 15.0, -5.0], [20.0, 0.0, 10.0]])
    _check(x, L_Box=10.0, linking_length=0.35, np_halo_min=2)


def test_list_with_skipped_regions():
    rng = np.random.default_rng(4)
    xs = [rng.normal(0, 0.3, (3, n)) + rng.uniform(50, 450, (3, 1)) for n in (5, 40, 1, 300, 9, 10, 1200)]
    _check(xs, L_Box=512.0, linking_length=0.1, np_halo_min=10)
