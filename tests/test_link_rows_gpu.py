"""Linking where the row, face and minimum-image rules change: one to seven
cells per axis, periodic, open and open along one axis only, sparse cells and
clumps (dense and very dense cells) in the middle and across the faces.
Partition and numbering equal to the oracle's."""
import numpy as np
import pytest

import py_fof_b200 as P
from tests.helpers import oracle_core

pytestmark = pytest.mark.gpu


def _points(rng, cells, extent, clump):
    n = cells ** 3 * 2
    x = rng.random((3, n)) * np.array(extent)[:, None]
    for c in range(clump):
        m = (40, 700, 90)[c]
        centre = np.array(extent) * ((0.5, 0.5, 0.5), (0.0, 0.99, 0.3), (1.0, 0.0, 0.0))[c]
        x = np.concatenate([x, centre[:, None] + 0.05 * extent[0] / cells * rng.standard_normal((3, m))], axis=1)
    return x[:, rng.permutation(x.shape[1])]


def _same(g, o):
    assert np.array_equal(g[0], o[0])
    assert np.array_equal(g[1], o[1])


@pytest.mark.parametrize("cells", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("shape", ["periodic", "open", "slab"])
@pytest.mark.parametrize("clump", [0, 1, 3])
def test_few_cells(cells, shape, clump):
    rng = np.random.default_rng(100 * cells + clump)
    L = 10.0
    box = {"periodic": (L, L, L), "open": (0.4 * L,) * 3, "slab": (L, 0.5 * L, L)}[shape]
    x = _points(rng, cells, box, clump)
    if shape == "periodic":
        x = np.mod(x, L)
    else:  # inside the box, away from its faces along the open axes
        x = np.mod(x + (0.2 * L if shape == "open" else 0.0), L)
    kw = dict(L_Box=L, linking_length=0.55 * box[0] / cells / 2 ** (1 / 3), np_halo_min=2, return_ang_mom=True)
    _same(P._fof_core(x, vp_list=np.zeros_like(x), **kw), oracle_core(x, vp_list=np.zeros_like(x), **kw))


def test_list_of_small_regions():
    """Many open regions of different sizes in one call."""
    rng = np.random.default_rng(5)
    xs = [_points(rng, 1 + k % 6, (2.0 + k % 3,) * 3, k % 4) + 20.0 for k in range(60)]
    vs = [np.zeros_like(x) for x in xs]
    kw = dict(vp_list=vs, L_Box=64.0, linking_length=0.2, np_halo_min=2, return_ang_mom=True)
    _same(P._fof_core(xs, **kw), oracle_core(xs, **kw))
