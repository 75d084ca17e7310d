"""Numbering of very many groups that share a cell: a knot far smaller than
the mean separation holds nearly all particles, each its own group (or in
pairs).  The ids are known: cells in order, then by first member.  The time
after the linking grows like the number of groups, not its square."""
import numpy as np
import pytest

import py_fof_b200 as P
from py_fof_b200 import _native

pytestmark = pytest.mark.gpu

L, SPAN = 3000.0, 900.0


def _knot(m, seed, pairs=False):
    """m^3 points (in pairs: twice as many), in the middle of one cell of a box
    that a particle at either corner stretches; shuffled."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(m, dtype=np.float64)] * 3, indexing="ij"), 0).reshape(3, -1)
    k = 0.01 * g + rng.uniform(-0.001, 0.001, g.shape)
    if pairs:
        k = np.concatenate([k, k + 0.001], axis=1)
    n = k.shape[1] + 2
    cell = (SPAN ** 3 / n) ** (1.0 / 3.0)
    mid = 10.0 + (np.floor(450.0 / cell) + 0.5) * cell
    assert 0.01 * m < 0.4 * cell
    k += mid - 0.005 * m
    x = np.concatenate([np.full((3, 1), 10.0), k, np.full((3, 1), 10.0 + SPAN)], axis=1)
    return x[:, np.concatenate([[0], 1 + rng.permutation(n - 2), [n - 1]])]


KW = dict(L_Box=L, linking_length=0.004)


# up to 1,024 candidates of one cell are numbered by counting, more by sorting
@pytest.mark.parametrize("m", [10, 11, 40])
def test_singles(m):
    x = _knot(m, m)
    n = x.shape[1]
    r = P._fof_core(x, np_halo_min=1, **KW)
    assert np.array_equal(r[1], np.arange(1, n + 1))


@pytest.mark.parametrize("m", [10, 11, 40])
def test_pairs(m):
    x = _knot(m, m, pairs=True)
    ids = P._fof_core(x, np_halo_min=2, **KW)[1]
    assert ids[0] == ids[-1] == 0
    mine = ids[1:-1]
    assert np.array_equal(np.bincount(mine)[1:], np.full(m ** 3, 2))
    _, first = np.unique(mine, return_index=True)
    assert np.all(np.diff(first) > 0)  # numbered by first member


def test_runs_above_and_below_the_line_in_one_call():
    """Two knots in cells of their own, and field groups, in one region."""
    a, b = _knot(14, 1), _knot(10, 2)
    x = np.concatenate([a[:, :-1], b[:, 1:-1] + 100.0, a[:, -1:]], axis=1)
    n = x.shape[1]
    rng = np.random.default_rng(3)
    p = np.concatenate([[0], 1 + rng.permutation(n - 2), [n - 1]])
    ids = P._fof_core(x[:, p], np_halo_min=1, **KW)[1]
    assert np.array_equal(np.sort(ids), np.arange(1, n + 1))
    na = a.shape[1] - 1
    for part in (ids[(p >= 1) & (p < na)], ids[(p >= na) & (p < n - 1)]):
        assert np.array_equal(part, np.arange(part[0], part[0] + part.size))


@pytest.mark.parametrize("order", [0, 1, 2])
def test_two_regions_and_cell_orders(order):
    """A list of two knots: the second's ids follow the first's, whatever the
    order inside the cells."""
    xs = [_knot(18, 5), _knot(11, 6)]
    with _native.options(cell_order=order):
        ids = P._fof_core(xs, np_halo_min=1, **KW)[1]
    assert np.array_equal(ids, np.arange(1, ids.size + 1))


def test_time_is_linear():
    ms = {}
    with _native.options(timing=1):
        for m in (40, 80):  # 64,000 and 512,000 groups
            x = _knot(m, m)
            t = []
            for _ in range(4):
                P._fof_core(x, np_halo_min=1, **KW)
                t.append(_native.last_stage_ms("after_link"))
            ms[m] = min(t)
    # eight times the groups: 8 if linear, 64 if quadratic
    assert ms[80] < 20 * ms[40], ms
