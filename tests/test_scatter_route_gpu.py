"""Both sides of the rule that sends a shuffled region through the two-step
scatter (16 bytes of output a particle against 64 MB: 4,000,000 particles),
with sizes that leave a partial tile: the same groups and ids as with the
reference's order inside the cells (option cell_order 1), which scatters
indices instead."""
import numpy as np
import pytest

import py_fof_b200 as P
from py_fof_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3999999, 4000000, 4000001, 4100003])
def test_same_ids_on_both_routes(n):
    rng = np.random.default_rng(n)
    L = 158.0
    x = rng.uniform(0, L, (3, n))
    x[:, : n // 8] = np.mod(x[:, n // 8: 2 * (n // 8)] + rng.normal(0, 0.05, (3, n // 8)), L)
    x = x[:, rng.permutation(n)]
    kw = dict(L_Box=L, linking_length=0.2, np_halo_min=3)
    a = P._fof_core(x, **kw)
    with _native.options(cell_order=1):
        b = P._fof_core(x, **kw)
    assert a[1].max() > 1000
    assert np.array_equal(a[1], b[1])
