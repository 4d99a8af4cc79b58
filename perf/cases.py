"""Performance cases of the forward path: what a user's program has it do, over the range of real sizes.

Kinds (``case["kind"]``), all through ``actfemtide_b200.forward``:

* ``tidal``: one step of a conductivity study on a resident mesh: new conductivities, assembly, the batched
  solve (1..16 systems: tidal periods x source patterns) and the fields at the sites.
* ``oneshot``: a forward from nothing but host arrays: mesh, numbering, pattern, assembly, solve, sites.
* ``packed``: independent uneven meshes in one packed solve (an ensemble of models).
* ``adjoint``: adjoint solves for site data and the sensitivities of every tetrahedron.
* ``mt``: the 3-D magnetotelluric forward (side faces, both polarisations, impedances).
* ``view``: plan-view evaluation of a solved batch on a grid of points.
* ``train``: loss and gradient of the learned preconditioner on residual samples.

Meshes are seeded synthetic boxes (``actfemtide_b200.synth``): uniform for the tidal kinds, graded for ``mt``.
Solves go to 1e-10 (5e-10 with the FP32 preconditioner), where the site fields are settled to about ten digits,
as difference quotients of an inversion need them.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from actfemtide_b200 import learned, synth
from actfemtide_b200.capi import xy_points
from actfemtide_b200.forward import Forward, MTForward

TOL = {"fp64": 1e-10, "pc32": 5e-10}
MT_TOL = 3e-12  # the impedances' small diagonal entries are a hundredth of the others
EXACT_EDGES = 24000  # dense complex LU of a mesh this size takes a second or two


def listed():
    return [
        # one station on a tiny mesh with the default solver (the reference's SSOR sweeps): start-up checks
        dict(name="ssor_4x4x6", kind="tidal", nx=4, ny=4, nz=6, half=10.0, ns=1, precond="SSOR", precision="fp64", nobs=1),
        # a single period on a small mesh: latency of every launch shows
        dict(name="tidal_12x12x9_1", kind="tidal", nx=12, ny=12, nz=9, ns=1, precond="HYBRID", precision="fp64", nobs=25),
        # ragged cell counts, two source patterns
        dict(name="tidal_23x17x13_2", kind="tidal", nx=23, ny=17, nz=13, ns=2, precond="HYBRID", precision="fp64", nobs=40),
        # the training mesh with the full batch (8 periods x 2 patterns), FP32 preconditioner
        dict(name="tidal_32x32x24_16", kind="tidal", nx=32, ny=32, nz=24, ns=16, precond="HYBRID", precision="pc32",
             nobs=25),
        # 8 periods of one pattern in full FP64 on the medium mesh
        dict(name="tidal_48x48x32_8", kind="tidal", nx=48, ny=48, nz=32, ns=8, precond="HYBRID", precision="fp64", nobs=400),
        # the full batch on a large mesh
        dict(name="tidal_56x56x40_16", kind="tidal", nx=56, ny=56, nz=40, ns=16, precond="HYBRID", precision="fp64",
             nobs=400),
        # the largest mesh, one period
        dict(name="tidal_88x88x56_1", kind="tidal", nx=88, ny=88, nz=56, ns=1, precond="HYBRID", precision="fp64", nobs=400),
        # a mesh seen for the first time: everything from host arrays
        dict(name="oneshot_32x32x24_4", kind="oneshot", nx=32, ny=32, nz=24, ns=4, precond="HYBRID", precision="pc32",
             nobs=100),
        # an ensemble of uneven meshes, one system each
        dict(name="packed_24", kind="packed", count=24, nmin=8, nmax=20, precision="pc32"),
        # sensitivities of 8 sites x 2 components
        dict(name="adjoint_14x14x11", kind="adjoint", nx=14, ny=14, nz=11, nobs=8),
        # magnetotelluric sounding, 4 frequencies x 2 polarisations
        dict(name="mt_20x20x20_4", kind="mt", nx=20, ny=20, nair=6, nearth=14, nf=4, nobs=36),
        # one training step's loss and gradient of the learned preconditioner
        dict(name="train_16x16x12", kind="train", nx=16, ny=16, nz=12, nsamp=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tidal"] * 6 + ["oneshot", "packed", "adjoint", "mt", "view", "train"])
    if kind in ("tidal", "oneshot", "view"):
        while True:
            nx = _log_int(rng, 7, 72)
            ny = max(6, int(nx * rng.uniform(0.7, 1.3)))
            nz = max(6, int(nx * rng.uniform(0.6, 1.0)))
            ns = rng.choice([1, 2, 4, 8, 16])
            limit = {"tidal": 6e6, "oneshot": 2e6, "view": 1e6}[kind]
            if edges(nx, ny, nz) * ns <= limit:
                break
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz, ns=ns, precond="HYBRID", precision=rng.choice(["fp64", "pc32"]),
                 nobs=_log_int(rng, 1, 400))
        if edges(nx, ny, nz) > 4e5:  # the FP32 preconditioner's attainable residual rises with the mesh
            c["precision"] = "fp64"
        if kind == "view":
            c["nobs"] = _log_int(rng, 900, 20000)
        if kind == "tidal" and rng.random() < 0.15:  # the reference's sweeps, on meshes they converge on
            c.update(nx=rng.randint(3, 5), ny=rng.randint(3, 5), nz=rng.randint(4, 8), half=10.0, precision="fp64",
                     precond=rng.choice(["SSOR", "SSOR_MC"]))
        return c
    if kind == "packed":
        lo = rng.randint(6, 10)
        return dict(kind=kind, count=rng.randint(2, 32), nmin=lo, nmax=lo + rng.randint(2, 12),
                    precision=rng.choice(["fp64", "pc32"]))
    if kind == "adjoint":
        n = _log_int(rng, 8, 18)
        return dict(kind=kind, nx=n, ny=max(6, n - rng.randint(0, 3)), nz=max(6, n - rng.randint(0, 4)),
                    nobs=rng.choice([1, 2, 4, 8]))
    if kind == "mt":
        n = _log_int(rng, 8, 26)
        return dict(kind=kind, nx=n, ny=max(6, n - rng.randint(0, 4)), nair=rng.randint(4, 8), nearth=rng.randint(8, 16),
                    nf=rng.choice([1, 2, 4, 8]), nobs=rng.randint(1, 100))
    n = _log_int(rng, 8, 24)
    return dict(kind=kind, nx=n, ny=n, nz=max(6, n - rng.randint(0, 6)), nsamp=rng.choice([1, 2, 4]))


# ----------------------------------------------------------------------------- inputs
def edges(nx, ny, nz):
    """Edges of a Kuhn-split box: axis edges, face diagonals, body diagonals."""
    return (nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
            + nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz)


@functools.lru_cache(maxsize=3)
def _box(nx, ny, nz, half):
    """The mesh of a uniform box and the hex of each land tetrahedron (the same for every seed)."""
    m = synth.tidal_box(nx, ny, nz, block=False, half_km=half, name=f"box{nx}x{ny}x{nz}")
    land = m.n4[m.tag >= 3] - 1
    cen = m.xyz[land].mean(axis=1)
    lo, hi = m.xyz.min(axis=0), m.xyz.max(axis=0)
    ijk = np.minimum(((cen - lo) / (hi - lo) * (nx, ny, nz)).astype(np.int64), (nx - 1, ny - 1, nz - 1))
    return m, (ijk[:, 0], ijk[:, 1], ijk[:, 2]), cen[:, 2] < -synth.SEA_DEPTH_KM


def _velocity(nodes_xyz, rng):
    """A rectilinear tidal current of 5 cm/s with a smooth modulation over the sea."""
    theta, phi, ph = rng.uniform(0, 2 * np.pi, 3)
    k = rng.uniform(-0.1, 0.1, 2)
    amp = 0.05 * (1 + 0.1 * np.sin(nodes_xyz[:, :2] @ k + ph)) * np.exp(1j * phi)
    v = np.zeros((len(nodes_xyz), 3), np.complex128)
    v[:, 0], v[:, 1] = amp * math.cos(theta), amp * math.sin(theta)
    return v


def _sites(nobs, rng, half=50.0):
    xy = rng.uniform(-0.84 * half, 0.84 * half, (nobs, 2))
    return np.stack([xy[:, 0], xy[:, 1], synth.surface_z(xy[:, 0], xy[:, 1]) - synth.SITE_DEPTH_KM], axis=1)


def _model(case, seed):
    """A seeded log-normal earth under sea and air on the case's box, with two source patterns and sites."""
    rng = np.random.default_rng(seed)
    dims = (case["nx"], case["ny"], case["nz"])
    base, ijk, sub = _box(*dims, case.get("half", 50.0))
    spacing = tuple(2 * base.bounds["xout"] / d for d in dims)
    logs = np.clip(-2.0 + synth.gaussian_random_field(dims, spacing, 8.0, rng), -4.0, 0.5)
    sigma = np.where(sub, 10.0 ** logs[ijk], synth.SIGMA_LAND)
    sources = [(base.F, _velocity(base.xyz[:base.nodes], rng)) for _ in range(2)]
    return dataclasses.replace(base, sigma_land=sigma, v=sources[0][1], sites=_sites(case["nobs"], rng, base.bounds["xout"])), sources


def _systems(ns):
    """8 tidal periods of the first pattern, then of the second; fewer systems: the first periods of both."""
    f = 1.0 / (3600.0 * np.array(synth.BATCH_PERIODS_H))
    half = ns if ns <= 1 else ns // 2
    src = np.zeros(ns, np.int32)
    src[half:] = 1
    return np.concatenate([f[:half], f[:ns - half]]), src


def prepare(case, seed):
    kind = case["kind"]
    if kind == "packed":
        parts = synth.uneven_models(case["count"], seed, case["nmin"], case["nmax"])
        fw = Forward(0)
        pk = synth.pack(parts)
        fw.load_packed(pk)
        sites = _sites(25, np.random.default_rng(seed))
        return dict(case=case, fw=fw, sigma=pk.sigma_tet, freqs=np.array([m.freqs[0] for m in parts]), sites=sites)
    if kind == "mt":
        rng = np.random.default_rng(seed)
        m = synth.mt_box(case["nx"], case["ny"], case["nair"], case["nearth"], ratio_air=1.2, ratio_earth=1.1, grf=True,
                         seed=seed, block_sigma=0.5)
        xy = rng.uniform(-35, 35, (case["nobs"], 2))
        sites = np.column_stack([xy, np.full(case["nobs"], -synth.SITE_DEPTH_KM)])
        fw = MTForward(0)
        fw.load_mt_model(m)
        return dict(case=case, fw=fw, freqs=np.logspace(-3, -1, 8)[-case["nf"]:], sites=sites)
    if kind == "train":
        m, _ = _model(dict(case, nobs=1), seed)
        fw = Forward(0)
        fw.load_model(m)
        fw.assemble()
        fw.mpnn_set_params(_net(seed))
        rng = np.random.default_rng(seed)
        # samples like right-hand sides and early residuals: confined to the free edges
        free = fw.export_system(float(m.freqs[0]))["bc"] == 0
        r = rng.standard_normal((case["nsamp"], fw.nline)) + 1j * rng.standard_normal((case["nsamp"], fw.nline))
        return dict(case=case, fw=fw, freq=float(m.freqs[0]), samples=r * free)
    m, sources = _model(case, seed)
    fw = Forward(0)
    s = dict(case=case, fw=fw, m=m, sources=sources, sites=m.sites)
    if kind == "oneshot":
        s["freqs"], s["srcs"] = _systems(case["ns"])
        return s
    fw.load_model(m, sources=sources)
    if kind == "tidal":
        s["freqs"], s["srcs"] = _systems(case["ns"])
    elif kind == "view":
        s["freqs"], s["srcs"] = _systems(case["ns"])
        fw.assemble()
        _solve(s)
        s["sites"] = _view_points(case, seed)
    elif kind == "adjoint":
        f = float(m.freqs[0])
        fw.assemble()
        fw.solve(f, precond="HYBRID", tol=1e-11)
        s.update(freq=f, x=fw.solution(0), rhs=fw.adjoint_sources(f, m.sites))
    return s


def _net(seed):
    """Weights of a network in training: the initial ones with a non-zero output layer."""
    p = learned.init_params(seed % 1000)
    p[-2 * learned.H:] = 0.05 * np.random.default_rng(seed).standard_normal(2 * learned.H)
    return p


def _view_points(case, seed):
    n = int(math.isqrt(case["nobs"]))
    dx, dy = np.random.default_rng(seed).uniform(0, 0.1, 2)
    return xy_points(-40.0 + dx, 40.0 + dx, -40.0 + dy, 40.0 + dy, n, n, -6.01)


def _solve(s):
    c = s["case"]
    r = s["fw"].solve(s["freqs"], s["srcs"], precond=c["precond"], precision=c["precision"], tol=TOL[c["precision"]])
    if not r.ok:
        raise RuntimeError(f"solve did not converge: {r}")


# ----------------------------------------------------------------------------- one pass
def run(s):
    case, fw = s["case"], s["fw"]
    kind = case["kind"]
    if kind in ("tidal", "oneshot"):
        m = s["m"]
        if kind == "oneshot":
            fw.load_model(m, sources=s["sources"])
        else:
            fw.set_cond(m.sigma_air, m.sigma_ocean, 1, sigma_file=m.sigma_land)
        fw.assemble()
        _solve(s)
        return fw.sites(s["sites"])
    if kind == "packed":
        fw.set_sigma(s["sigma"])
        fw.assemble()
        r = fw.solve(s["freqs"], precond="HYBRID", precision=case["precision"], tol=TOL[case["precision"]])
        if not r.ok:
            raise RuntimeError(f"packed solve did not converge: {r}")
        return fw.sites(s["sites"])
    if kind == "adjoint":
        nadj = s["rhs"].shape[1]
        r = fw.solve_rhs(np.full(nadj, s["freq"]), s["rhs"], precond="HYBRID", tol=1e-9)
        if not r.ok:
            raise RuntimeError(f"adjoint solve did not converge: {r}")
        return fw.jacobian(s["freq"], s["x"], nadj)
    if kind == "mt":
        r = fw.mt_forward(s["freqs"], s["sites"], precond="HYBRID", tol=MT_TOL)
        if not r.solve.ok:
            raise RuntimeError(f"MT solve did not converge: {r.solve}")
        return dict(be=r.be, z=r.z, rho=r.rho, pha=r.pha)
    if kind == "view":
        return fw.sites_grid(s["sites"])
    loss, grad = fw.mpnn_loss_grad(s["freq"], s["samples"])
    return dict(loss=loss, grad=grad)


# ----------------------------------------------------------------------------- floor
def work(case):
    """The matrix written and read once, the systems' right-hand sides and solutions once each, and one product
    with the matrix per system: no solver does with less."""
    kind = case["kind"]
    if kind == "packed":
        n = case["count"] * edges(*[(case["nmin"] + case["nmax"]) // 2] * 3) * 3 // 4
        ns = 1
    elif kind == "mt":
        n, ns = edges(case["nx"], case["ny"], case["nair"] + case["nearth"]), 2 * case["nf"]
    else:
        n = edges(case["nx"], case["ny"], case["nz"])
        ns = case.get("ns", 2 * case.get("nobs", 0) if kind == "adjoint" else case.get("nsamp", 1))
    nnz = 16.25 * n
    if kind == "view":
        return {"bytes": 16.0 * n * ns + case["nobs"] * (24 + 80.0 * ns), "flops": 5 * 48.0 * case["nobs"] * ns}
    if kind == "train":  # forward and backward through 6 layers of width 48: features and gradients in BF16
        return {"bytes": ns * n * 6 * 4 * 96.0 + 20.0 * nnz, "flops": ns * n * 6 * 3 * 2 * 144 * 48.0}
    out = 16.0 * ns * (0.86 * n if kind == "adjoint" else 5.0 * case.get("nobs", 25))
    return {"bytes": 40.0 * nnz + 32.0 * n * ns + out, "flops": 8.0 * nnz * ns}


# ----------------------------------------------------------------------------- 64-bit answers without the library
KL = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))  # local edges (node pairs) of a tetrahedron
MU0 = 4e-7 * math.pi
KM = 1e3


def _elements(m, dev):
    """Edge numbering and Whitney elements in FP64: global edge ids, signs, gradients, volumes, Dirichlet edges."""
    n4 = torch.as_tensor(m.n4, device=dev).long() - 1
    xyz = torch.as_tensor(m.xyz, device=dev, dtype=torch.float64)
    a, b = n4[:, [k for k, _ in KL]], n4[:, [l for _, l in KL]]
    key, eid = torch.unique(torch.minimum(a, b) * len(xyz) + torch.maximum(a, b), return_inverse=True)
    sgn = torch.where(a < b, 1.0, -1.0).double()
    p = xyz[n4]
    J = p[:, 1:] - p[:, :1]
    g = torch.linalg.inv(J).transpose(1, 2)
    grad = torch.cat([-g.sum(1, keepdim=True), g], 1)      # gradients of the barycentric coordinates
    vol = torch.linalg.det(J).abs() / 6
    e0, e1 = xyz[key // len(xyz)], xyz[key % len(xyz)]
    bd = m.bounds
    out = torch.zeros(len(key), dtype=torch.bool, device=dev)
    for c, lo, hi in ((0, -bd["xout"], bd["xout"]), (1, -bd["yout"], bd["yout"]), (2, bd["zmin"], bd["zmax"])):
        out |= (e0[:, c] <= lo + 1) & (e1[:, c] <= lo + 1)
        out |= (e0[:, c] >= hi - 1) & (e1[:, c] >= hi - 1)
    return xyz, n4, eid, sgn, grad, vol, out


def _mass(grad, vol, sgn):
    """Element matrices of w_i . w_j and of curl w_i . curl w_j, with the edges' global signs."""
    gg = grad @ grad.transpose(1, 2)
    lam = (1 + torch.eye(4, dtype=torch.float64, device=vol.device)) / 20
    Y = torch.stack([torch.stack([lam[k, m] * gg[:, l, n] - lam[k, n] * gg[:, l, m] - lam[l, m] * gg[:, k, n]
                                  + lam[l, n] * gg[:, k, m] for m, n in KL], -1) for k, l in KL], 1)
    curl = 2 * torch.stack([torch.linalg.cross(grad[:, k], grad[:, l]) for k, l in KL], 1)
    w = (sgn[:, :, None] * sgn[:, None, :]) * vol[:, None, None]
    return Y * w, (curl @ curl.transpose(1, 2)) * w, curl


def _dense(m, el, freq, sigma):
    _, _, eid, sgn, grad, vol, out = el
    Y, S, _ = _mass(grad, vol, sgn)
    n = len(out)
    val = S.to(torch.complex128) + 2j * math.pi * freq * MU0 * KM * KM * sigma[:, None, None] * Y
    A = torch.zeros(n * n, dtype=torch.complex128, device=vol.device)
    A.index_add_(0, (eid[:, :, None] * n + eid[:, None, :]).reshape(-1), val.reshape(-1))
    A = A.view(n, n)
    A[out] = 0
    A[:, out] = 0
    A[out, out] = 1
    return A


def _source(m, el, sigma, F, v):
    _, n4, eid, sgn, grad, vol, out = el
    dev = vol.device
    vF = torch.zeros(len(m.xyz), 3, dtype=torch.complex128, device=dev)
    vF[:m.nodes] = torch.linalg.cross(torch.as_tensor(v, device=dev), torch.as_tensor(F, device=dev).to(torch.complex128))
    q = vF[n4]                                              # (t, node, 3)
    gq = torch.einsum("tlc,tjc->tlj", grad.to(torch.complex128), q)
    lam = ((1 + torch.eye(4, dtype=torch.float64, device=dev)) / 20).to(torch.complex128)
    S2 = torch.stack([gq[:, l] @ lam[k] - gq[:, k] @ lam[l] for k, l in KL], 1)
    sea = torch.as_tensor(m.tag, device=dev) == 2
    S2 = S2 * (sgn * (vol * sigma * sea * MU0 * 1e3)[:, None])
    b = torch.zeros(len(out), dtype=torch.complex128, device=dev)
    b.index_add_(0, eid.reshape(-1), S2.reshape(-1))
    b[out] = 0
    return b


def _site_rows(el, sites):
    """Per site its tetrahedron's edges and the values of w and curl w there."""
    xyz, n4, eid, sgn, grad, vol, _ = el
    ids, w, c = [], [], []
    for x in torch.as_tensor(sites, device=vol.device, dtype=torch.float64):
        lam = torch.einsum("tlc,tc->tl", grad, x - xyz[n4[:, 0]])
        lam[:, 0] += 1
        t = int(lam.amin(1).argmax())
        ids.append(eid[t])
        w.append(torch.stack([lam[t, k] * grad[t, l] - lam[t, l] * grad[t, k] for k, l in KL]) * sgn[t][:, None])
        c.append(2 * torch.stack([torch.linalg.cross(grad[t, k], grad[t, l]) for k, l in KL]) * sgn[t][:, None])
    return torch.stack(ids), torch.stack(w), torch.stack(c)


def exact(case, seed):
    """Dense LU in complex FP64 of a separately assembled system, for the meshes it is quick for."""
    kind = case["kind"]
    if kind not in ("tidal", "oneshot", "view", "adjoint") or edges(case["nx"], case["ny"], case["nz"]) > EXACT_EDGES:
        return None
    if kind == "view" and case["nobs"] > 2500 or case.get("ns", 1) > 8:
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    m, sources = _model(case, seed)
    el = _elements(m, dev)
    sigma = torch.as_tensor(m.sigma_per_tet(), device=dev)
    sites = _view_points(case, seed) if kind == "view" else m.sites
    ids, w, c = _site_rows(el, sites)
    w, c = w.to(torch.complex128), c.to(torch.complex128)
    if kind == "adjoint":
        f = float(m.freqs[0])
        n = len(el[6])
        C = torch.zeros(n, len(sites), 2, dtype=torch.complex128, device=dev)
        for s_ in range(len(sites)):
            C[ids[s_], s_] = -2j * math.pi * f * w[s_, :, :2]
        C = C.reshape(n, -1)                                # Dirichlet rows of A are the identity
        b = _source(m, el, sigma, *sources[0])
        X = torch.linalg.solve(_dense(m, el, f, sigma), torch.cat([b[:, None], C], 1))
        Y = _mass(el[4], el[5], el[3])[0].to(torch.complex128)
        live = (~el[6])[el[2]].to(torch.complex128)
        wx = torch.einsum("tij,tj->ti", Y, X[el[2], 0] * live) * live
        J = -2j * math.pi * f * MU0 * KM * KM * torch.einsum("tik,ti->kt", X[el[2], 1:], wx) * sigma
        return J.cpu().numpy()
    freqs, srcs = _systems(case["ns"])
    res = np.zeros((case["ns"], 5, len(sites)), np.complex128)
    rhs = [_source(m, el, sigma, F, v) for F, v in sources]
    for f in sorted(set(freqs)):
        ks = [k for k in range(case["ns"]) if freqs[k] == f]
        X = torch.linalg.solve(_dense(m, el, f, sigma), torch.stack([rhs[srcs[k]] for k in ks], 1))
        for i, k in enumerate(ks):
            x = X[:, i][ids]
            B = torch.einsum("sj,sjc->cs", x, c)
            E = -2j * math.pi * f * torch.einsum("sj,sjc->cs", x, w)[:2]
            res[k] = torch.cat([B, E]).cpu().numpy()
    return res
