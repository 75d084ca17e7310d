"""FP32 short-range sums of chunks that a whole block adds up: the sums stay
compensated across the block's warps.

A knot of 2,000 light members sits 0.002 from one heavy member; the light
ones together are three units in the last place of the heavy one's potential,
each warp's share of them less than half a unit, so an uncompensated addition
of the warps' sums loses them.  The potentials with the light masses are
compared with those of the same positions with the light masses 0, where only
the heavy member's term is left, identically rounded; the difference is known
in 64 bits.

Tolerance, in units of the last place of the potentials, on the mean over the
knot: both calls round unbiasedly (the compensated sum and the final
additions, each at most half a unit either way, over 2,000 targets), so the
mean of the difference is within half a unit of the exact one; the long-range
part, a hundredth of the total, changes by 3e-7 of itself.  An uncompensated
addition loses one to three units."""
import numpy as np
import pytest

from py_fof_b200 import _native

pytestmark = pytest.mark.gpu

S15 = 15 * 0.67 * 512 / 300.0
EPS = 1e-6
SPACING = 0.125  # of a 48^3 grid, span 2.0
A_VAL = 6.0 * 3.141592653589793238462643383279502884197  # the factor a / (6 pi) is 1


def _depth(r, h):
    e = 2.0 * r / h
    inner = (208.0 - e ** 2 * (112.0 + e ** 2 * (-56.0 + e * (14.0 + e * (8.0 - 3.0 * e))))) / (70.0 * h)
    with np.errstate(divide="ignore"):
        outer = (128.0 - (e ** 2 * (448.0 + e * (-280.0 + e * (56.0 + e * (14.0 + e * (-8.0 + e))))) - 224.0 * e
                          - 12.0 / e)) / (70.0 * h)
        return np.where(r >= h, 1.0 / r, np.where(e <= 1.0, inner, outer))


def test_compensated_across_warps():
    n, R = 2000, 0.002
    rng = np.random.default_rng(3)
    d = rng.standard_normal((3, n))
    d *= 0.1 * R / np.linalg.norm(d, axis=0)
    q = np.empty((3, n + 3), np.float32)
    q[:, 0] = 0.0  # the heavy member
    q[:, 1:n + 1] = d + np.array([R, 0.0, 0.0])[:, None]
    q[:, n + 1] = [1.0, 1.0, 1.0]
    q[:, n + 2] = [-1.0, -1.0, -1.0]
    knot = slice(1, n + 1)
    x = q[:, knot].astype(np.float64)
    r_heavy = np.linalg.norm(x - q[:, :1], axis=0)
    rr = np.linalg.norm(x[:, :, None] - x[:, None, :], axis=0)
    np.fill_diagonal(rr, 1.0)
    term = _depth(rr, EPS) - _depth(rr, 3.5 * SPACING)
    np.fill_diagonal(term, 0.0)
    heavy = _depth(r_heavy, EPS) - _depth(r_heavy, 3.5 * SPACING)
    # the heavy potential near 2^8 (1.2 of it, so a unit is 2^-15), the light
    # sum three units
    w_heavy = np.float32(1.2 * 2.0 ** 8 / heavy.mean())
    unit = 2.0 ** (8 - 23)
    w_light = np.float32(3.0 * unit / term.sum(1).mean())
    w = np.zeros(n + 3, np.float32)
    w[0] = w_heavy
    w[n + 1:] = 1e-12
    base, g0 = _native.halo_potential(q, w, softening=EPS, a_val=A_VAL, s15=S15, fp64=False)
    w[knot] = w_light
    full, g1 = _native.halo_potential(q, w, softening=EPS, a_val=A_VAL, s15=S15, fp64=False)
    assert g0 == g1 == 1
    base, full = base[knot].astype(np.float64), full[knot].astype(np.float64)
    assert np.all((-base > 2.0 ** 8) & (-full < 2.0 ** 9))
    got = (full - base) / unit
    want = -float(w_light) * term.sum(1) / unit
    assert abs(float((got - want).mean())) < 0.5, (got.mean(), want.mean())
