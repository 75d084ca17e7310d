"""Softening 0: the short-range residual is 1/r minus the split kernel, on
plain and refined particle-mesh halos, both precisions.  First-pass potentials
against the CPU oracle (tolerance as in test_pm_gpu.py: 1e-5 of the halo's
largest |phi|), and whole calls; coincident members, whose 1/r is infinite,
are refused."""
import numpy as np
import pytest

from oracle import oracle as O
from py_fof_b200 import _native

pytestmark = pytest.mark.gpu

S15 = 15 * 0.67 * 512 / 300.0


def _lattice_ball(n, step, seed, centre=(0.0, 0.0, 0.0)):
    """n points of a jittered lattice around `centre`: no pair closer than step / 2."""
    m = int(np.ceil((2 * n) ** (1.0 / 3.0))) + 1
    g = np.stack(np.meshgrid(*[np.arange(m) - 0.5 * (m - 1)] * 3, indexing="ij"), 0).reshape(3, -1)
    g = g[:, np.argsort((g ** 2).sum(0), kind="stable")[:n]]
    rng = np.random.default_rng(seed)
    x = step * (g + rng.uniform(-0.25, 0.25, g.shape)) + np.asarray(centre)[:, None]
    return x[:, rng.permutation(n)]


def _cases():
    yield "plain", _lattice_ball(1500, 0.06, 1)
    rng = np.random.default_rng(2)
    yield "refined", np.concatenate([_lattice_ball(16000, 0.02, 3, (0.1, 0.2, -0.3)), rng.uniform(-5, 5, (3, 400))],
                                    axis=1)


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("softening", [0.0, 1e-42])
@pytest.mark.parametrize("name,x", list(_cases()), ids=[c[0] for c in _cases()])
def test_first_pass_potential(name, x, softening, fp64):
    n = x.shape[1]
    q = (x - x[:, :1]).astype(np.float32)
    w = np.random.default_rng(n).lognormal(-0.045, 0.3, n).astype(np.float32)
    xv = np.zeros((n, 6), np.float32)
    xv[:, :3] = q.T
    g_o, phi_o = O.first_potential(xv, w, np.arange(1, n + 1), softening=softening, a_val=1.0, s15=S15)
    assert np.all(np.isfinite(phi_o))
    phi, g = _native.halo_potential(q, w, softening=softening, fp64=fp64, s15=S15)
    assert g == g_o > 0
    if name == "refined":
        assert _native.get_stat("refined_regions") > 0
    assert np.abs(phi - phi_o).max() < 1e-5 * np.abs(phi_o).max()


@pytest.mark.parametrize("fp64", [1, 0])
def test_whole_call(fp64):
    x = _lattice_ball(1500, 0.06, 5) + 50.0
    n = x.shape[1]
    args = (x, np.zeros_like(x), None, np.array([n], np.int32), 1, 100.0, 0.2, 10, 1, 0)
    with _native.options(unbind_fp64=fp64):
        r = _native.run(*args, 0.0, 1.0, 0.0, S15, 0, n)
    assert r[3] == 0 and r[0].all()  # cold: every member is bound


@pytest.mark.parametrize("fp64", [True, False])
def test_coincident_members_are_refused(fp64):
    x = _lattice_ball(1500, 0.06, 7)
    x[:, 900] = x[:, 30]
    q = (x - x[:, :1]).astype(np.float32)
    with pytest.raises(RuntimeError):
        _native.halo_potential(q, np.ones(1500, np.float32), softening=0.0, fp64=fp64, s15=S15)
