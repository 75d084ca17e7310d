"""Convolutions at the transform length that a halo's box asks for: boxes on
both sides of the steps between lengths, on the 64, 128 and 256 grids.
First-pass potentials against the CPU oracle, which transforms the whole grid
(tolerance as in test_pm_gpu.py: 1e-5 of the halo's largest |phi|), and the
bytes of the passes, which tell the length."""
import itertools

import numpy as np
import pytest

from oracle import oracle as O
from py_fof_b200 import _native

pytestmark = pytest.mark.gpu

S15 = 15 * 0.67 * 512 / 300.0
# members, extent, lengths that may be chosen (the box is a few nodes wider
# than the extent over the spacing)
CASES = [(1300, 3.7, {48}), (1300, 7.2, {64}),
         (1100, 8.0, {96}), (1100, 12.0, {108}), (1100, 15.2, {128}),
         (20100, 3.0, {128}), (20100, 4.1, {144}), (20100, 4.7, {160}), (20100, 5.3, {180}),
         (20100, 5.7, {192}), (20100, 6.3, {216}), (20100, 7.2, {240}), (20100, 7.75, {256})]


@pytest.mark.parametrize("n,extent,lengths", CASES)
def test_potential_at_length(n, extent, lengths):
    rng = np.random.default_rng(n)
    x = rng.random((3, n)) * extent
    x[:, 1] = 0.0  # both corners of the box are occupied
    x[:, 2] = extent * (1 - 1e-6)
    q = (x - x[:, :1]).astype(np.float32)
    w = rng.lognormal(-0.045, 0.3, n).astype(np.float32)
    xv = np.zeros((n, 6), np.float32)
    xv[:, :3] = q.T
    g_o, phi_o = O.first_potential(xv, w, np.arange(1, n + 1), softening=0.1, a_val=1.0, s15=S15)
    before = _native.get_stat("pm_fft_bytes")  # (of this process's potentials so far)
    phi, g = _native.halo_potential(q, w, fp64=True, s15=S15)
    assert g == g_o > 0
    err = np.abs(phi - phi_o).max() / np.abs(phi_o).max()
    assert err < 1e-5, err
    # bytes of the five passes (conv_bytes) for a box of sx x sy x sz nodes,
    # a cube but for the rounding of its corners
    got = _native.get_stat("pm_fft_bytes") - before
    sizes = set()
    for m in (48, 64, 96, 108, 128, 144, 160, 180, 192, 216, 240, 256):
        for s in range(3, m // 2 + 2):
            for sx, sy, sz in itertools.product((s, s - 1), repeat=3):
                if got == 16 * sx * sy * sz + 64 * (m // 2 + 1) * (sy + m) * sz:
                    sizes.add(m)
    assert sizes & lengths, (g, got, sizes, lengths)
