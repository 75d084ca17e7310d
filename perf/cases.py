"""Performance cases: the calls that users of py_fof_b200 make.

Three entry points are measured, each the way a program calls it:

* ``fof`` / ``fof_with_info`` on NumPy arrays: the reference's own API, host
  inputs and host results, through the whole call;
* ``pyfof_run_device`` (``_native.run_device``) on inputs in device memory:
  simulation codes and pipelines that hold their particles on the GPU;
* ``pyfof_halo_potential`` (``_native.halo_potential``): the potential of one
  halo.

Inputs follow the recipes of ``workloads.py`` (Plummer box, NFW list,
lognormal box), generated with torch on the GPU from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import py_fof_b200 as P
from py_fof_b200 import _native

LINK = 0.2          # linking length in units of the mean particle separation
SOFT = 0.1
G_CODE = 1.0 / (6.0 * math.pi)
S15_BOX = 15.0 * 0.67 * 256.0 / 300.0    # span limit of the boxes (cube units)
S15_LIST = 15.0 * 0.67 * 512.0 / 300.0   # span limit of lists and single regions
MEAN_DENSITY = 2_000_000 / (4.0 / 3.0 * math.pi * (0.45 * S15_LIST) ** 3)  # inside R_vir, NFW lists


def listed():
    return [
        # one small cut-out around a group, a call per object in a loop: pure latency
        {"name": "region_fof_2k", "kind": "region", "n": 2000, "bound": False},
        # unbinding of one small halo in physical units (direct summation): latency again
        {"name": "halo_unbind_900", "kind": "region", "n": 900, "bound": True},
        # a small periodic test box, FoF only, through the NumPy API
        {"name": "box_fof_64_host", "kind": "box_host", "n": 64 ** 3, "bound": False},
        # a periodic box with unbinding through the NumPy API (copies included)
        {"name": "box_unbind_128_host", "kind": "box_host", "n": 128 ** 3, "bound": True},
        # a halo catalogue of a list of cut-outs with unbinding (fof_with_info)
        {"name": "list_info_1k_host", "kind": "list_host", "halos": 1000, "mmax": 50_000},
        # the potential of one group-sized halo (particle mesh, 256^3 grid)
        {"name": "potential_30k", "kind": "potential", "n": 30_000, "fp64": True},
        # FoF only of a simulation-sized box held on the device, x[i][3] layout, an odd size
        {"name": "box_fof_251_dev", "kind": "box_dev", "n": 251 ** 3, "bound": False, "fp64": True, "aos": True},
        # the headline workload: FoF + unbinding of a 256^3 box held on the device
        {"name": "box_unbind_256_dev", "kind": "box_dev", "n": 256 ** 3, "bound": True, "fp64": True, "aos": False},
        # the same stage on the FP32 product path, a smaller box of an odd size
        {"name": "box_unbind_203_fp32_dev", "kind": "box_dev", "n": 203 ** 3, "bound": True, "fp64": False,
         "aos": False},
        # batched unbinding of 20,000 isolated halos (20 members to a million)
        {"name": "list_unbind_20k_dev", "kind": "list_dev", "halos": 20_000, "mmax": 2_000_000, "fp64": True},
        # one zoom region: a massive cluster with substructure, few large candidates
        {"name": "zoom_unbind_1m_dev", "kind": "zoom", "n": 1_000_000, "fp64": True},
        # FoF of a large clustered box, 768^3 particles in snapshot (spatial) order
        {"name": "lognormal_fof_768_dev", "kind": "lognormal", "n": 768 ** 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["region", "region", "box_host", "list_host", "potential", "box_dev", "box_dev", "list_dev",
                       "zoom", "lognormal"])
    if kind == "region":
        bound = rng.random() < 0.5
        return {"kind": kind, "n": _log_int(rng, 100, 20_000), "bound": bound}
    if kind == "box_host":
        return {"kind": kind, "n": _log_int(rng, 20_000, 128 ** 3), "bound": rng.random() < 0.5}
    if kind == "list_host":
        return {"kind": kind, "halos": _log_int(rng, 20, 1000), "mmax": _log_int(rng, 500, 50_000)}
    if kind == "potential":
        return {"kind": kind, "n": _log_int(rng, 100, 60_000), "fp64": rng.random() < 0.5}
    if kind == "box_dev":
        return {"kind": kind, "n": _log_int(rng, 64 ** 3, 256 ** 3), "bound": rng.random() < 0.6,
                "fp64": rng.random() < 0.6, "aos": rng.random() < 0.4}
    if kind == "list_dev":
        return {"kind": kind, "halos": _log_int(rng, 200, 20_000), "mmax": _log_int(rng, 20_000, 2_000_000),
                "fp64": rng.random() < 0.6}
    if kind == "zoom":
        return {"kind": kind, "n": _log_int(rng, 50_000, 1_000_000), "fp64": rng.random() < 0.6}
    return {"kind": kind, "n": _log_int(rng, 2_000_000, 768 ** 3)}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _directions(g, n):
    d = _randn(g, 3, n)
    return d / d.norm(dim=0)


def _power_law(n, mmin, mmax, slope=-1.9):
    """n member counts at the quantiles of dN/dM ~ M^slope (the same for
    every seed, so that a case's work does not vary with it)."""
    e = slope + 1.0
    u = (np.arange(n) + 0.5) / n
    return np.maximum(mmin, np.floor((mmin ** e + u * (mmax ** e - mmin ** e)) ** (1.0 / e))).astype(np.int64)


def _virial(g, sigma, kick_frac=0.1):
    """Isotropic velocities of dispersion sigma, a tenth of them kicked."""
    n = sigma.numel()
    v = _randn(g, 3, n) * sigma
    kick = _rand(g, n) < kick_frac
    return v + torch.where(kick, 3.0 * sigma, torch.zeros_like(sigma)) * _directions(g, n)


def _plummer_box(n, seed, velocities):
    """Uniform background and Plummer spheres on a jittered lattice in a
    periodic box of unit mean density, shuffled (workloads.plummer_box)."""
    g = _gen(seed)
    side = n ** (1.0 / 3.0)
    n_halos = max(1, round(n / 4096))
    n_h = int(0.3 * n)
    c = _power_law(n_halos, 20, 5000).astype(np.float64)
    counts = np.maximum(1, np.floor(c * (n_h / c.sum()))).astype(np.int64)
    n_h = int(counts.sum())
    per = math.ceil(n_halos ** (1.0 / 3.0) - 1e-9)
    spacing = side / per
    cell = torch.arange(per ** 3, device="cuda")[torch.argsort(_rand(g, per ** 3))[:n_halos]]
    cells = torch.stack([cell % per, (cell // per) % per, cell // (per * per)]).double()
    centres = (cells + 0.5 + 0.25 * (_rand(g, 3, n_halos) - 0.5)) * spacing
    owner = torch.repeat_interleave(torch.arange(n_halos, device="cuda"), torch.as_tensor(counts, device="cuda"))
    a = 1.5
    u = _rand(g, n_h).clamp(1e-12, 1 - 1e-9)
    r = a / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    xp = torch.cat([_rand(g, 3, n - n_h) * side, centres[:, owner] + r * _directions(g, n_h)], dim=1)
    perm = torch.argsort(_rand(g, n))
    xp = torch.remainder(xp, side)[:, perm].contiguous()
    if not velocities:
        return xp, None, None, side
    m = torch.as_tensor(counts, device="cuda").double()[owner]
    sigma = torch.sqrt(G_CODE * m / (6.0 * torch.sqrt(r * r + a * a)))
    vh = _virial(g, sigma) + (3.0 * _randn(g, 3, n_halos))[:, owner]
    vp = torch.cat([_randn(g, 3, n - n_h), vh], dim=1)[:, perm].contiguous()
    mp = torch.exp(0.3 * _randn(g, n) - 0.045)
    return xp, vp, mp, side


def _nfw(g, sizes, centres):
    """NFW spheres of fixed mean density, one after the other: positions and
    virial velocities (workloads.nfw_halos)."""
    sizes_t = torch.as_tensor(sizes, device="cuda")
    nh = len(sizes)
    owner = torch.repeat_interleave(torch.arange(nh, device="cuda"), sizes_t)
    rv = (sizes_t.double() / (4.0 / 3.0 * math.pi * MEAN_DENSITY)) ** (1.0 / 3.0)
    conc = 5.0 + 10.0 * _rand(g, nh)
    mu = lambda x: torch.log1p(x) - x / (1.0 + x)  # noqa: E731
    c = conc[owner]
    n = owner.numel()
    target = _rand(g, n) * mu(c)
    lo, hi = torch.zeros_like(c), c.clone()
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        f = mu(mid) < target
        lo, hi = torch.where(f, mid, lo), torch.where(f, hi, mid)
    x = 0.5 * (lo + hi)
    m = sizes_t.double()[owner]
    r = x * (rv / conc)[owner]
    pos = centres[:, owner] + r * _directions(g, n)
    sigma = torch.sqrt(G_CODE * (m * mu(x) / mu(c)).clamp(min=1.0) / r.clamp(min=0.05) / 3.0)
    return pos, _virial(g, sigma)


def _nfw_list(halos, mmax, seed):
    g = _gen(seed)
    sizes = _power_law(halos, 20, mmax)[np.random.default_rng(seed).permutation(halos)]
    xp, vp = _nfw(g, sizes, 100.0 + 300.0 * _rand(g, 3, halos))
    return xp.contiguous(), vp.contiguous(), sizes.astype(np.int32)


def _lognormal_box(n, seed):
    """Poisson sample of a lognormal density field (P(k) ~ k^-2, sigma 1.5)
    on a mesh of two mean separations, in mesh order (workloads.lognormal_box)."""
    g = _gen(seed)
    side = n ** (1.0 / 3.0)
    mesh = max(16, 2 * round(side / 4))
    f = torch.randn(mesh, mesh, mesh, generator=g, device="cuda")
    fk = torch.fft.rfftn(f)
    k = torch.fft.fftfreq(mesh, device="cuda")
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + torch.fft.rfftfreq(mesh, device="cuda")[None, None, :] ** 2
    k2[0, 0, 0] = float("inf")
    f = torch.fft.irfftn(fk * k2 ** -0.5, s=(mesh, mesh, mesh)).double().reshape(-1)
    del fk, k2
    w = torch.exp(f * (1.5 / f.std()) - 1.125)
    lam = w * ((n - 6.0 * math.sqrt(n)) / w.sum())
    del f, w
    counts = torch.poisson(lam, generator=g).long()
    del lam
    total = int(counts.sum())
    xp = torch.empty(3, n, device="cuda", dtype=torch.float64)
    h = side / mesh
    m = min(total, n)
    ends = torch.cumsum(counts, 0)
    step = 1 << 22
    p0 = 0
    for c0 in range(0, counts.numel(), step):
        c1 = min(counts.numel(), c0 + step)
        cell = torch.repeat_interleave(torch.arange(c0, c1, device="cuda"), counts[c0:c1])
        p1 = min(int(ends[c1 - 1]), m)
        cell = cell[:p1 - p0]
        for d, j in enumerate((cell % mesh, (cell // mesh) % mesh, cell // (mesh * mesh))):
            xp[d, p0:p1] = torch.remainder((j + _rand(g, p1 - p0)) * h, side)
        p0 = p1
    if m < n:  # the few left over go anywhere
        xp[:, m:] = _rand(g, 3, n - m) * side
    return xp, side


def _zoom(n, seed):
    """A cluster (an NFW sphere with bound subhaloes) and its thin surroundings."""
    g = _gen(seed)
    n_sub = max(8, n // 20_000)
    subs = _power_law(n_sub, max(100, n // 2000), max(400, n // 20), slope=-1.8)
    main = int(0.95 * n) - int(subs.sum())
    rv = (main / (4.0 / 3.0 * math.pi * MEAN_DENSITY)) ** (1.0 / 3.0)
    centres = torch.zeros(3, n_sub + 1, device="cuda", dtype=torch.float64)
    centres[:, 1:] = 0.6 * rv * _rand(g, n_sub) ** 0.5 * _directions(g, n_sub)
    x, v = _nfw(g, np.concatenate([[main], subs]), centres)
    left = n - x.shape[1]
    x = torch.cat([x, 40.0 * (_rand(g, 3, left) - 0.5)], dim=1) + 256.0
    v = torch.cat([v, _randn(g, 3, left)], dim=1)
    perm = torch.argsort(_rand(g, n))
    return x[:, perm].contiguous(), v[:, perm].contiguous()


def _region(n, seed):
    """A halo, a few smaller companions and field particles around them."""
    g = _gen(seed)
    parts = [max(20, int(f * n)) for f in (0.5, 0.15, 0.1)]
    centres = torch.zeros(3, 3, device="cuda", dtype=torch.float64)
    centres[0] = torch.tensor([0.0, 9.0, -9.0])
    x, v = _nfw(g, np.array(parts), centres)
    left = max(0, n - x.shape[1])
    x = torch.cat([x, 24.0 * (_rand(g, 3, left) - 0.5)], dim=1)[:, :n] + 256.0
    v = torch.cat([v, 0.5 * _randn(g, 3, left)], dim=1)[:, :n]
    perm = torch.argsort(_rand(g, n))
    return x[:, perm].contiguous(), v[:, perm].contiguous()


def _host(t):
    return None if t is None else t.cpu().numpy()


# the physical units of the single-region unbinding calls (a 300 Mpc/h box of 512^3 particles)
PHYS = {"units": "physical", "L_Box": 300.0, "n_sim": 512 ** 3, "linking_length": LINK * 300.0 / 512.0,
        "softening": SOFT * 300.0 / 512.0}


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "region":
        x, v = _region(case["n"], seed)
        if case["bound"]:  # Mpc/h and km/s
            v = v / (512.0 / (150.0 * math.sqrt(0.3) * 300.0))
            x = x * (300.0 / 512.0)
        s.update(xp=_host(x), vp=_host(v))
    elif kind == "box_host":
        x, v, m, side = _plummer_box(case["n"], seed, case["bound"])
        s.update(xp=_host(x), vp=_host(v), mp=_host(m), side=side)
    elif kind == "list_host":
        x, v, sizes = _nfw_list(case["halos"], case["mmax"], seed)
        cuts = np.cumsum(sizes)[:-1]
        s.update(xp=[np.ascontiguousarray(p) for p in np.split(_host(x), cuts, axis=1)],
                 vp=[np.ascontiguousarray(p) for p in np.split(_host(v), cuts, axis=1)])
    elif kind == "potential":
        g = _gen(seed)
        x, _ = _nfw(g, np.array([case["n"]]), torch.zeros(3, 1, device="cuda", dtype=torch.float64))
        q = (x - x[:, :1]).float()
        w = torch.exp(0.3 * _randn(g, case["n"]) - 0.045).float()
        s.update(q=_host(q), w=_host(w))
    else:
        v = m = None
        if kind == "box_dev":
            x, v, m, side = _plummer_box(case["n"], seed, case["bound"])
            np_halo, s15, bound = np.array([case["n"]], np.int32), S15_BOX, case["bound"]
        elif kind == "lognormal":
            x, side = _lognormal_box(case["n"], seed)
            np_halo, s15, bound = np.array([case["n"]], np.int32), S15_BOX, False
        elif kind == "list_dev":
            x, v, np_halo = _nfw_list(case["halos"], case["mmax"], seed)
            side, s15, bound = 512.0, S15_LIST, True
        else:
            x, v = _zoom(case["n"], seed)
            side, s15, bound, np_halo = 512.0, S15_LIST, True, np.array([case["n"]], np.int32)
        n = x.shape[1]
        if case.get("aos"):
            x = x.t().contiguous()
            v = None if v is None else v.t().contiguous()
        s.update(xp=x, vp=v, mp=m, np_halo=np_halo, n=n, side=side, s15=s15, bound=bound,
                 in_halo=torch.zeros(n, dtype=torch.int32, device="cuda"),
                 halo_id=torch.zeros(n, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------- passes

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "region":
        if case["bound"]:
            return P.fof(s["xp"], s["vp"], bound_check=True, return_ang_mom=True, **PHYS)
        return P.fof(s["xp"], s["vp"], return_ang_mom=True)
    if kind == "box_host":
        return P.fof(s["xp"], s["vp"], L_Box=s["side"], linking_length=LINK, np_halo_min=20, mp_list=s["mp"],
                     bound_check=case["bound"], softening=SOFT, ng_global=256.0, return_ang_mom=True)
    if kind == "list_host":
        r = P.fof_with_info(s["xp"], s["vp"], L_Box=512.0, linking_length=LINK, bound_check=True, softening=SOFT,
                            return_ang_mom=True)
        # the catalogue as arrays of fixed length (a region holds about one halo)
        counts = np.zeros(r["in_halo"].size, np.int64)
        counts[:r["nhalo_found"]] = r["np_per_halo"]
        members = np.full(r["in_halo"].size, -1, np.int64)
        if r["nhalo_found"]:
            np.concatenate(r["halo_indices"], out=members[:counts.sum()])
        return r["in_halo"], counts, members, r["ang_mom"]
    if kind == "potential":
        phi, _ = _native.halo_potential(s["q"], s["w"], softening=SOFT, s15=S15_LIST, fp64=case["fp64"])
        return phi
    ptr = lambda t: 0 if t is None else t.data_ptr()  # noqa: E731
    args = (ptr(s["xp"]), ptr(s["vp"]), ptr(s["mp"]),
            _native.LAYOUT_AOS if case.get("aos") else _native.LAYOUT_SOA, s["np_halo"], len(s["np_halo"]), s["n"],
            s["side"], LINK, 20 if kind == "box_dev" else 10, int(s["bound"]), 0, SOFT, 1.0, 0.0, s["s15"], 0,
            s["in_halo"].data_ptr(), s["halo_id"].data_ptr())
    if case.get("fp64", True):
        ang_mom, ierr = _native.run_device(*args)
    else:
        with _native.options(unbind_fp64=0):
            ang_mom, ierr = _native.run_device(*args)
    if ierr:
        raise RuntimeError(f"ierr={ierr}: {_native.last_error()}")
    return s["in_halo"], s["halo_id"], ang_mom


def work(case):
    """Each input read once and each output written once."""
    kind = case["kind"]
    if kind == "region":
        return {"bytes": 49 * case["n"], "flops": 0}
    if kind == "box_host":
        return {"bytes": (57 if case["bound"] else 25) * case["n"], "flops": 0}
    if kind == "list_host":
        return {"bytes": 61 * int(_power_law(case["halos"], 20, case["mmax"]).sum()), "flops": 0}
    if kind == "potential":
        return {"bytes": 20 * case["n"], "flops": 0}
    if kind == "box_dev":
        return {"bytes": (64 if case["bound"] else 32) * case["n"], "flops": 0}
    if kind == "lognormal":
        return {"bytes": 32 * case["n"], "flops": 0}
    n = case["n"] if kind == "zoom" else int(_power_law(case["halos"], 20, case["mmax"]).sum())
    return {"bytes": 56 * n, "flops": 0}


# ------------------------------------------------------------- 64-bit results

def _depth(r, h):
    """The spline-softened 1/r (bound_fortran.f90:3080-3102)."""
    e = 2.0 * r / h
    inner = (208.0 - e * e * (112.0 + e * e * (-56.0 + e * (14.0 + e * (8.0 - 3.0 * e))))) / (70.0 * h)
    es = e.clamp(min=1e-12)
    prim = es * es * (448.0 + es * (-280.0 + es * (56.0 + es * (14.0 + es * (-8.0 + es))))) - 224.0 * es - 12.0 / es
    outer = (128.0 - prim) / (70.0 * h)
    return torch.where(e <= 1.0, inner, torch.where(r < h, outer, 1.0 / r.clamp(min=1e-300)))


def exact(case, seed):
    if case["kind"] == "potential":
        s = prepare(case, seed)
        q = torch.as_tensor(s["q"], device="cuda").double()
        w = torch.as_tensor(s["w"], device="cuda").double()
        n = case["n"]
        phi = torch.empty(n, device="cuda", dtype=torch.float64)
        step = max(1, (1 << 25) // n)
        for i in range(0, n, step):
            d = (q[:, i:i + step, None] - q[:, None, :]).pow(2).sum(0).sqrt()
            t = _depth(d, SOFT) * w
            t[torch.arange(t.shape[0], device="cuda"), torch.arange(i, i + t.shape[0], device="cuda")] = 0.0
            phi[i:i + step] = -G_CODE * t.sum(1)
        return phi
    if case["kind"] == "region" and not case["bound"]:
        # groups by brute force, then the groups' angular momentum about their centres
        s = prepare(case, seed)
        x = torch.as_tensor(s["xp"], device="cuda")
        v = torch.as_tensor(s["vp"], device="cuda")
        n = x.shape[1]
        label = torch.arange(n, device="cuda")
        step = max(1, (1 << 26) // n)
        linked = torch.cat([(x[:, i:i + step, None] - x[:, None, :]).pow(2).sum(0) <= LINK * LINK
                            for i in range(0, n, step)])
        while True:
            new = torch.cat([torch.where(linked[i:i + step], label, n).amin(1) for i in range(0, n, step)])
            new = new[new]
            if torch.equal(new, label):
                break
            label = new
        size = torch.bincount(label, minlength=n)
        am = torch.zeros(3, device="cuda", dtype=torch.float64)
        for h in torch.nonzero(size >= 10).reshape(-1).tolist():
            k = label == h
            dx = x[:, k] - x[:, k].mean(1, keepdim=True)
            dv = v[:, k] - v[:, k].mean(1, keepdim=True)
            am += torch.linalg.cross(dx, dv, dim=0).sum(1)
        return None, am.reshape(3, 1).cpu().numpy()
    # memberships are whole numbers, and the angular momentum of a bound or
    # large set is a sum over members that only the whole method gives
    return None
