"""The short-range residual at the edges of its chunking: cells and bricks
with one to many chunks, chunks just below and above the size summed by a
whole block, a halo one cell wide, refined halos with targets of all three
cutoffs, and pairs far inside the softening length.  First-pass potentials
against the CPU oracle; tolerance as in test_pm_gpu.py (1e-5 of the halo's
largest |phi|: the oracle's own FP32 grid weights and FFT)."""
import numpy as np
import pytest

from oracle import oracle as O
from py_fof_b200 import _native

pytestmark = pytest.mark.gpu

S15 = 15 * 0.67 * 512 / 300.0


def _ball(n, radius, seed, centre=(0.0, 0.0, 0.0)):
    rng = np.random.default_rng(seed)
    d = rng.standard_normal((3, n))
    d *= radius * rng.random(n) ** (1.0 / 3.0) / np.linalg.norm(d, axis=0)
    return d + np.asarray(centre)[:, None]


def _cases():
    rng = np.random.default_rng(5)
    yield "ball_1023", _ball(1023, 0.15, 1)
    yield "ball_1024", _ball(1024, 0.15, 2)
    yield "ball_1500", _ball(1500, 0.4, 3)
    yield "rod", np.stack([rng.uniform(-5, 5, 1501), rng.normal(0, 0.01, 1501), rng.normal(0, 0.01, 1501)])
    x = _ball(1200, 0.3, 4)
    x[:, 600:] = x[:, :600] + 1e-4 * rng.standard_normal((3, 600))  # pairs at about 1e-3 of the softening
    yield "close_pairs", x
    # spacing 0.125 (span above 7.8), a clump refined by 4, a smaller one by 2, thin surroundings
    yield "refined", np.concatenate([_ball(16000, 0.35, 6, (0.1, 0.2, -0.3)), _ball(5000, 0.3, 7, (3.1, 0.5, 0.0)),
                                     rng.uniform(-5, 5, (3, 1500))], axis=1)


@pytest.mark.parametrize("name,x", list(_cases()), ids=[c[0] for c in _cases()])
def test_first_pass_potential(name, x):
    n = x.shape[1]
    q = (x - x[:, :1]).astype(np.float32)
    w = np.random.default_rng(n).lognormal(-0.045, 0.3, n).astype(np.float32)
    xv = np.zeros((n, 6), np.float32)
    xv[:, :3] = q.T
    g_o, phi_o = O.first_potential(xv, w, np.arange(1, n + 1), softening=0.1, a_val=1.0, s15=S15)
    scale = np.abs(phi_o).max()
    for fp64 in (True, False):
        phi, g = _native.halo_potential(q, w, fp64=fp64, s15=S15)
        assert g == g_o > 0
        if name == "refined":
            assert _native.get_stat("refined_regions") > 1
        err = np.abs(phi - phi_o).max() / scale
        assert err < 1e-5, (fp64, err)
