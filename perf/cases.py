"""The work that users of this framework have it do, as measurable cases.

The framework steps Lagrangian parcels through a cell-valued carrier velocity and hands the
momentum source back to the fluid solver.  A case is one pass of such a program:

  step     a coupled fluid time step (or a few of them) of a solver that lives on the GPU: the new
           cell velocity goes in, `steps` parcel steps run, the source comes out on the device
  clouds   the same for a handle with many independent clouds (one source each)
  tet      the same on a tetrahedral mesh (parcels are tracked by a face walk)
  noalloc  the allocation-free step on caller-owned arrays (st_step_noalloc)
  host     a coupled fluid time step of a solver on the host: U from host memory, source back to it
  readback steps between two outputs of a run, then the parcels and owning cells to the host
  adjoint  the time-averaged source and its pull-back (an optimisation step)

Physics: water droplets in air (Schiller-Naumann or Stokes drag, explicit or implicit Euler),
dt = 1e-4 s, a 0.1 m box with reflecting walls, a Taylor-Green-like carrier, lognormal diameters
around 20 um clipped to [8, 60] um, parcels in flight with 70 to 100 % of the carrier's velocity.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "scale-track_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import scaletrack as st  # noqa: E402

RHO_P, RHO_F, MU_F = 1000.0, 1.2, 1.8e-5
DT, L = 1e-4, 0.1
DEV = "cuda"


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: a few thousand parcels on caller-owned arrays, latency and launches
        dict(name="noalloc_hex12_3e3", kind="noalloc", nx=12, ny=12, nz=12, parcels=3001,
             drag="stokes_implicit", substeps=1),
        # the allocation-free step at its largest mesh
        dict(name="noalloc_hex64_1e6", kind="noalloc", nx=64, ny=64, nz=64, parcels=1_000_003,
             drag="schiller_naumann", substeps=1),
        # the reference's own settings (FP32, Stokes implicit, ten substeps) on a cavity of its
        # tutorial's size: a small coupled step, bound by launches
        dict(name="step_hex20_fp32_stokes", kind="step", nx=20, ny=20, nz=20, parcels=10_000,
             precision="fp32", drag="stokes_implicit", substeps=10, deposit="deterministic",
             sort=0, steps=1, u_bytes=4),
        # the FP64 configuration of 1e5 parcels on 32^3 cells, a ragged count
        dict(name="step_hex32_fp64", kind="step", nx=32, ny=32, nz=32, parcels=100_001,
             precision="fp64", drag="schiller_naumann", substeps=1, deposit="deterministic",
             sort=0, steps=4, u_bytes=8),
        # an ordinary box with odd sizes, FP64 with the atomic deposit, U of a float32 solver
        dict(name="step_hex97_fp64_atomic", kind="step", nx=97, ny=64, nz=53,
             parcels=2_000_003, precision="fp64", drag="schiller_naumann", substeps=1,
             deposit="atomic", sort=20, steps=4, u_bytes=4),
        # the headline configuration: 1e7 parcels on 128^3 cells, mixed precision, one re-sort
        # cycle of 20 steps with a time-varying carrier
        dict(name="step_hex128_mixed", kind="step", nx=128, ny=128, nz=128,
             parcels=10_000_000, precision="mixed", drag="schiller_naumann", substeps=1,
             deposit="deterministic", sort=20, steps=20, u_bytes=4),
        # 64 clouds of log-uniform sizes on one 64^3 mesh, ten substeps per step
        dict(name="clouds64_hex64_mixed", kind="clouds", nx=64, ny=64, nz=64, clouds=64,
             size_min=1_000, size_max=2_000_000, size_seed=2, precision="mixed",
             drag="schiller_naumann", substeps=10, sort=0, steps=1, u_bytes=4),
        # a small tet mesh in FP64 with two substeps
        dict(name="tet12_fp64", kind="tet", n=12, parcels=50_001, precision="fp64",
             drag="schiller_naumann", substeps=2, sort=10, steps=2, u0=3.0),
        # the tet configuration: 5.3e6 tets, 2e7 parcels, one re-sort cycle of ten steps
        dict(name="tet96_mixed", kind="tet", n=96, parcels=20_000_000, precision="mixed",
             drag="schiller_naumann", substeps=1, sort=10, steps=10, u0=3.0),
        # a fluid solver on the host: U (double) up, one step, the source (double) down
        dict(name="host_hex64_mixed", kind="host", nx=64, ny=64, nz=64, parcels=1_000_000,
             precision="mixed", drag="schiller_naumann", substeps=1, sort=20, u_bytes=8),
        # four steps and an output of a run: parcels and owning cells back on the host
        dict(name="readback_hex64_fp32", kind="readback", nx=64, ny=64, nz=64,
             parcels=1_000_000, precision="fp32", drag="stokes_implicit", substeps=2, sort=20,
             steps=4),
        # the adjoint configuration: 200 steps of 1e6 parcels, checkpoints every 20
        dict(name="adjoint_hex128_mixed", kind="adjoint", nx=128, ny=128, nz=128,
             parcels=1_000_000, precision="mixed", steps=200, checkpoint=20, sort=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "clouds", "tet", "tet", "noalloc",
                       "noalloc", "host", "readback", "adjoint"])
    drag = rng.choice(["schiller_naumann", "schiller_naumann", "stokes_implicit"])
    sub = rng.choice([1, 1, 1, 2, 5, 10])
    prec = rng.choice(["mixed", "mixed", "fp64", "fp32"])
    box = {k: _log(rng, 8, 128) for k in ("nx", "ny", "nz")}
    if kind == "step":
        return dict(kind=kind, **box, parcels=_log(rng, 1_000, 5_000_000), precision=prec,
                    drag=drag, substeps=sub,
                    deposit=rng.choice(["deterministic", "deterministic", "atomic"]),
                    sort=rng.choice([0, 10, 20]), steps=rng.choice([1, 2, 4]),
                    u_bytes=rng.choice([4, 8]))
    if kind == "clouds":
        return dict(kind=kind, nx=rng.randint(8, 64), ny=rng.randint(8, 64),
                    nz=rng.randint(8, 64), clouds=rng.randint(2, 40),
                    size_min=_log(rng, 100, 2_000), size_max=_log(rng, 10_000, 1_000_000),
                    size_seed=rng.randint(0, 1000), precision=prec, drag=drag, substeps=sub,
                    sort=rng.choice([0, 20]), steps=rng.choice([1, 2]),
                    u_bytes=rng.choice([4, 8]))
    if kind == "tet":
        return dict(kind=kind, n=_log(rng, 6, 64), parcels=_log(rng, 1_000, 6_000_000),
                    precision=rng.choice(["mixed", "mixed", "fp64"]), drag=drag,
                    substeps=rng.choice([1, 1, 2, 4]), sort=rng.choice([0, 10]),
                    steps=rng.choice([1, 2, 4]), u0=rng.choice([1.0, 3.0]))
    if kind == "noalloc":
        return dict(kind=kind, nx=_log(rng, 6, 64), ny=_log(rng, 6, 64), nz=_log(rng, 6, 64),
                    parcels=_log(rng, 500, 2_000_000), drag=drag, substeps=sub)
    if kind == "host":
        return dict(kind=kind, **{k: _log(rng, 8, 72) for k in box},
                    parcels=_log(rng, 1_000, 2_000_000), precision=prec, drag=drag,
                    substeps=sub, sort=rng.choice([0, 20]), u_bytes=rng.choice([4, 8]))
    if kind == "readback":
        return dict(kind=kind, **{k: _log(rng, 8, 72) for k in box},
                    parcels=_log(rng, 1_000, 1_500_000), precision=prec, drag=drag,
                    substeps=sub, sort=rng.choice([0, 20]), steps=rng.choice([1, 4]))
    return dict(kind=kind, **box, parcels=_log(rng, 1_000, 800_000),
                precision=rng.choice(["mixed", "mixed", "fp64"]), steps=rng.choice([20, 50, 130]),
                checkpoint=rng.choice([7, 10, 20]), sort=rng.choice([0, 20]))


def fluid_factor(k):
    """Time-varying carrier: the factor on U in step k of a pass."""
    return 1.0 + 0.2 * math.sin(2.0 * math.pi * (k + 3) * DT / 0.05)


# ------------------------------------------------------------------------------ the inputs
def _gen(seed, stream=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * (seed + 1) + stream)
    return g


def _tgv(x, y, z, u0):
    a, b, c = math.pi / L * x, math.pi / L * y, math.pi / L * z
    return torch.stack([u0 * torch.sin(a) * torch.cos(b) * torch.cos(c),
                        -u0 * torch.cos(a) * torch.sin(b) * torch.cos(c),
                        torch.zeros_like(a)])


def _carrier(points, seed, u0):
    """[m, 3] FP64 carrier velocity at the cell centres [3, m]: the analytic field with one
    per cent of noise (a resolved solver's field differs from cell to cell)."""
    u = _tgv(points[0], points[1], points[2], u0)
    u = u + 0.01 * u0 * torch.randn(u.shape, generator=_gen(seed, 1), device=DEV,
                                    dtype=torch.float64)
    return u.t().contiguous()


def _hex_centres(c):
    k, j, i = torch.meshgrid(*[(torch.arange(c[a], device=DEV, dtype=torch.float64) + 0.5)
                               * (L / c[a]) for a in ("nz", "ny", "nx")], indexing="ij")
    return torch.stack([i.reshape(-1), j.reshape(-1), k.reshape(-1)])


def _parcels(n, seed, u0=1.0, stream=2, d_median=20e-6):
    """Positions and velocities [3, n] and diameters [n], FP64, values that FP32 velocities and
    diameters hold exactly."""
    g = _gen(seed, stream)
    x = torch.rand((3, n), generator=g, device=DEV, dtype=torch.float64) * (L * (1 - 1e-6))
    v = _tgv(x[0], x[1], x[2], u0) * (0.7 + 0.3 * torch.rand((1, n), generator=g, device=DEV,
                                                             dtype=torch.float64))
    d = d_median * torch.exp(0.3 * torch.randn(n, generator=g, device=DEV, dtype=torch.float64))
    d = d.clamp(8e-6, 60e-6)
    return x, v.float().double(), d.float().double()


def _cloud_sizes(c):
    rng = np.random.default_rng(c["size_seed"])
    sizes = np.exp(rng.uniform(np.log(c["size_min"]), np.log(c["size_max"]), c["clouds"]))
    return sizes.astype(np.int64), rng.uniform(15e-6, 40e-6, c["clouds"])


_MESHES = {}


def _tet_mesh(n):
    """n^3 hexes of the box, each split into six tets around a diagonal (conforming), hexes in
    Morton order, inner vertices jittered by 15 % of the spacing (walls stay planar).  Returns
    vertices [nv, 3], tets and neighbours [nt, 4] and the Morton rank of each lattice hex."""
    if n in _MESHES:
        return _MESHES[n]
    _MESHES.clear()
    h = L / n
    ar = torch.arange(n + 1, device=DEV)
    vk, vj, vi = torch.meshgrid(ar, ar, ar, indexing="ij")
    ijk = torch.stack([vi.reshape(-1), vj.reshape(-1), vk.reshape(-1)], 1)
    g = torch.Generator(device=DEV)
    g.manual_seed(1)
    jit = (torch.rand(ijk.shape, generator=g, device=DEV, dtype=torch.float64) * 2 - 1) * 0.15 * h
    jit[(ijk == 0) | (ijk == n)] = 0.0
    verts = ijk.double() * h + jit
    hk, hj, hi = torch.meshgrid(ar[:n], ar[:n], ar[:n], indexing="ij")
    hexes = torch.stack([hi.reshape(-1), hj.reshape(-1), hk.reshape(-1)], 1)
    code = torch.zeros(n ** 3, device=DEV, dtype=torch.int64)
    for b in range(10):
        for a in range(3):
            code |= ((hexes[:, a] >> b) & 1) << (3 * b + a)
    order = torch.argsort(code)
    rank = torch.empty_like(order)
    rank[order] = torch.arange(n ** 3, device=DEV)
    hexes = hexes[order]
    cube = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
    corner = torch.stack([((hexes[:, 2] + o[2]) * (n + 1) + hexes[:, 1] + o[1]) * (n + 1)
                          + hexes[:, 0] + o[0] for o in cube], 1)
    split = ((0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6), (0, 5, 1, 6))
    tets = torch.stack([corner[:, list(s)] for s in split], 1).reshape(-1, 4)
    faces = torch.stack([tets[:, [k for k in range(4) if k != f]] for f in range(4)], 1)
    faces = faces.reshape(-1, 3).sort(dim=1).values
    key = (faces[:, 0] * (n + 1) ** 3 + faces[:, 1]) * (n + 1) ** 3 + faces[:, 2]
    key, at = key.sort()
    same = key[1:] == key[:-1]
    a, b = at[:-1][same], at[1:][same]
    nbr = torch.full((tets.shape[0] * 4,), -1, device=DEV, dtype=torch.int64)
    nbr[a], nbr[b] = b // 4, a // 4
    _MESHES[n] = (verts, tets.int(), nbr.reshape(-1, 4).int(), rank)
    return _MESHES[n]


def _tet_hint(x, n, rank):
    """The first tet of the lattice hex that holds each parcel, where its walk starts."""
    i = (x * (n / L)).long().clamp(0, n - 1)
    return (6 * rank[(i[2] * n + i[1]) * n + i[0]]).int()


class _OnDevice:
    """A handle's device array for torch; keeps the handle alive as long as the tensor."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False),
                                             version=3, strides=None)


def _view(h, cloud, ncells):
    return torch.as_tensor(_OnDevice(h, h.source_device_ptr(cloud), (ncells, 3)), device=DEV)


def _params(c, **kw):
    return st.params(mu_c=MU_F, rho_c=RHO_F, rho_d=RHO_P, drag_model=c.get("drag", "sn_explicit"),
                     precision=c.get("precision", "mixed"), n_substeps=c.get("substeps", 1),
                     sort_interval=c.get("sort", 0), **kw)


def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind == "tet":
        verts, tets, nbr, rank = _tet_mesh(c["n"])
        mesh = st.tet_mesh_desc(_host(verts), _host(tets), _host(nbr), 0.0, L)
        centres = verts[tets.long()].mean(1).t()
        u0 = c["u0"]
    else:
        mesh = st.mesh_desc((c["nx"], c["ny"], c["nz"]), 0.0, L)
        centres, u0 = _hex_centres(c), 1.0
    U = _carrier(centres, seed, u0)
    ncells = U.shape[0]
    del centres
    vdt = torch.float64 if c.get("precision") == "fp64" else torch.float32
    s["fs"] = [fluid_factor(k) for k in range(c.get("steps", 1))]
    if kind == "noalloc":
        x, v, d = _parcels(c["parcels"], seed)
        s["prm"], s["mesh"] = _params(c), mesh
        s["x"] = [x[a].clone() for a in range(3)]
        s["v"] = [v[a].float() for a in range(3)]
        s["d"], s["U"] = d.float(), U.float()
        s["source"] = torch.zeros((ncells, 3), device=DEV, dtype=torch.float64)
        torch.cuda.synchronize()
        return s
    kw = dict(deposit=c.get("deposit", "deterministic"), n_clouds=c.get("clouds", 1))
    h = s["h"] = st.ParcelTracker(_params(c, **kw), mesh, device=0)
    if kind == "clouds":
        for i, (m, dm) in enumerate(zip(*_cloud_sizes(c))):
            x, v, d = _parcels(int(m), seed, stream=2 + i, d_median=float(dm))
            h.set_parcels(_host(x), _host(v), _host(d), cloud=i)
    else:
        x, v, d = _parcels(c["parcels"], seed, u0)
        hint = _host(_tet_hint(x, c["n"], rank)) if kind == "tet" else None
        h.set_parcels(_host(x), _host(v), _host(d), hint=hint)
    if kind == "host":
        s["U"] = _host(U if c["u_bytes"] == 8 else U.float())
    elif kind in ("readback", "adjoint"):
        h.set_fluid_velocity(_host(U.to(vdt)))
        if kind == "adjoint":
            # the cotangent of a squared distance to a target field has the source's smoothness
            s["cot"] = _host(_carrier(_hex_centres(c), seed + 77, 1.0))
    else:
        eb = c.get("u_bytes", 8 if vdt == torch.float64 else 4)
        s["U"], s["eb"] = U if eb == 8 else U.float(), eb
        s["source"] = [_view(h, i, ncells) for i in range(c.get("clouds", 1))]
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------------------- one pass
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "noalloc":
        p = ctypes.c_void_p
        rc = st.lib().st_step_noalloc(
            ctypes.byref(s["prm"]), ctypes.byref(s["mesh"]), c["parcels"],
            *[p(t.data_ptr()) for t in s["x"]], *[p(t.data_ptr()) for t in s["v"]],
            p(s["d"].data_ptr()), p(s["U"].data_ptr()), p(s["source"].data_ptr()), DT, s["fs"][0],
            p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(st.last_error())
        return {"source": s["source"], "x": s["x"], "v": s["v"]}
    h = s["h"]
    if kind == "host":
        h.set_fluid_velocity(s["U"])
        h.step(DT, s["fs"][0])
        return {"source": h.get_source(dtype=s["U"].dtype)}
    if kind == "readback":
        for f in s["fs"]:
            h.step(DT, f)
        x, v, d = h.get_parcels()
        return {"x": x, "v": v, "d": d, "cells": h.get_cells()}
    if kind == "adjoint":
        a = (c["steps"], c["checkpoint"], DT, s["fs"])
        S = h.mean_source_forward(*a)
        dalpha, dscale, dv0 = h.mean_source_pullback(s["cot"], *a)
        return {"mean": S, "dalpha": dalpha, "dscale": dscale, "dv0": dv0}
    h.set_fluid_velocity_device(s["U"].data_ptr(), s["eb"])
    for f in s["fs"]:
        h.step(DT, f)
    h.source_device_ptr(0)   # orders the handle's stream after the source
    return {"source": s["source"]}


# ---------------------------------------------------------------------------- what it needs
def work(case):
    """Bytes: per step the parcel state read (with diameters, and the owning tet) and written,
    U read and the FP64 source written once per cell, and a tet's FP64 face planes and
    neighbours; host and adjoint passes add their own inputs and outputs."""
    c, kind = case, case["kind"]
    if kind == "tet":
        cells = 6 * c["n"] ** 3
    else:
        cells = c["nx"] * c["ny"] * c["nz"]
    n = int(_cloud_sizes(c)[0].sum()) if kind == "clouds" else c["parcels"]
    steps, sub = c.get("steps", 1), c.get("substeps", 1)
    prec = c.get("precision", "mixed")
    per = {"mixed": 76, "fp64": 104, "fp32": 52}[prec]
    vb = 8 if prec == "fp64" else 4
    if kind == "tet":
        by = steps * (n * (per + 8) + cells * (3 * vb + 24 + 128 + 16))
    elif kind == "adjoint":
        # checkpoints written and read, state, cotangent and mean source once, dv0
        nseg = -(-steps // c["checkpoint"])
        by = n * (per // 2 + 24 + nseg * 2 * (24 + 3 * vb)) + cells * (3 * vb + 48)
        return {"bytes": float(by), "flops": float(n) * steps * 350.0}
    elif kind == "readback":
        by = steps * (n * per + cells * 36) + n * (56 + 4)
    else:
        by = steps * (n * per + cells * 3 * vb + c.get("clouds", 1) * cells * 24)
    return {"bytes": float(by), "flops": float(n) * steps * sub * 90.0}


# ------------------------------------------------------------------------------ in 64 bits
def _drag(c, du, f, d):
    """g: dv = g du of Schiller-Naumann drag"""
    re = du.norm(dim=0) * d * (RHO_F / MU_F)
    return f * (1.0 + 0.15 * re ** 0.687)


class _Hex:
    def __init__(self, c):
        self.n = torch.tensor([c["nx"], c["ny"], c["nz"]], device=DEV)[:, None]
        self.rd = 1.0 / (L / self.n.double())

    def cell(self, x, _old=None):
        i = torch.floor(x * self.rd).long()
        return (i[2] * self.n[1] + i[1]) * self.n[0] + i[0]

    def wall(self, x):
        i = torch.floor(x * self.rd).long()
        return (i < 0) | (i >= self.n)


class _Tet:
    def __init__(self, c):
        verts, tets, nbr, _ = _tet_mesh(c["n"])
        self.nbr = nbr.long()
        planes = []
        for f in range(4):
            p, q, r = (verts[tets[:, k].long()] for k in range(4) if k != f)
            nrm = torch.linalg.cross(q - p, r - p)
            away = ((verts[tets[:, f].long()] - p) * nrm).sum(1, keepdim=True)
            nrm = torch.where(away > 0, -nrm, nrm)
            planes.append(torch.cat([nrm, (nrm * p).sum(1, keepdim=True)], 1))
        self.planes = torch.stack(planes, 1)

    def cell(self, x, old):
        cell = old.clone()
        at = torch.arange(x.shape[1], device=DEV)
        for _ in range(200):
            pl, y = self.planes[cell[at]], x[:, at].t()
            s, f = ((pl[:, :, :3] * y[:, None, :]).sum(2) - pl[:, :, 3]).max(1)
            to = self.nbr[cell[at], f]
            go = (s > 0) & (to >= 0)
            at = at[go]
            if not at.numel():
                break
            cell[at] = to[go]
        return cell

    def wall(self, x):
        return (x < 0) | (x > L)


def _exact_step(c, geo, x, v, d, U, cell, factor, ncells):
    """One step of `substeps` substeps in 64 bits: new x, v, cell and the source [ncells, 3]."""
    sub = c.get("substeps", 1)
    dt = DT / sub
    m = RHO_P / RHO_F * math.pi * d ** 3 / 6.0
    f = 18.0 * MU_F * dt / (RHO_P * d * d)
    S = torch.zeros((ncells, 3), device=DEV, dtype=torch.float64)
    start, here = v.clone(), cell
    for t in range(sub):
        u = U[here].t() * factor
        if c["drag"] == "stokes_implicit":
            vn = (v + f * u) / (1.0 + f)
        else:
            vn = v + _drag(c, u - v, f, d) * (u - v)
        xn = x + vn * dt
        b = geo.wall(xn)
        start = torch.where(b, start - 2 * v, start)
        xn, vn = torch.where(b, x, xn), torch.where(b, -v, vn)
        cell = geo.cell(xn, cell)
        if t + 1 < sub:
            moved = cell != here
            dep = torch.where(moved, m * (start - vn), torch.zeros_like(vn))
            S.index_add_(0, here, dep.t())
            start = torch.where(moved, vn, start)
            here = cell
        x, v = xn, vn
    S.index_add_(0, here, (m * (start - v)).t())
    return x, v, cell, S


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "tet":
        verts, tets, _, rank = _tet_mesh(c["n"])
        geo, u0 = _Tet(c), c["u0"]
        centres = verts[tets.long()].mean(1).t()
    else:
        geo, u0, centres = _Hex(c), 1.0, _hex_centres(c)
    U = _carrier(centres, seed, u0)
    ncells = U.shape[0]
    if c.get("precision") != "fp64" or c.get("u_bytes") == 4:
        U = U.float().double()   # what the framework is given, or holds
    if kind == "adjoint":
        return _exact_adjoint(c, seed, geo, U, ncells)
    if kind == "clouds":
        sets = [_parcels(int(m), seed, stream=2 + i, d_median=float(dm))
                for i, (m, dm) in enumerate(zip(*_cloud_sizes(c)))]
    else:
        sets = [_parcels(c["parcels"], seed, u0)]
    out = []
    for x, v, d in sets:
        if c.get("precision") == "fp32":
            x = x.float().double()
        cell = geo.cell(x, _tet_hint(x, c["n"], rank).long() if kind == "tet" else None)
        for k in range(c.get("steps", 1)):
            x, v, cell, S = _exact_step(c, geo, x, v, d, U, cell, fluid_factor(k), ncells)
        out.append(S)
    if kind == "noalloc":
        return {"source": S, "x": [x[a] for a in range(3)], "v": [v[a] for a in range(3)]}
    if kind == "readback":
        return {"x": x, "v": v, "d": d, "cells": None}
    return {"source": S} if kind == "host" else {"source": out}


def _exact_adjoint(c, seed, geo, U, ncells):
    """The mean source and its pull-back with cells and bounces frozen, by reverse-mode
    differentiation of every step."""
    x, v, d = _parcels(c["parcels"], seed)
    T = c["steps"]
    one = torch.ones((), device=DEV, dtype=torch.float64)
    S = torch.zeros((ncells, 3), device=DEV, dtype=torch.float64)
    G = _carrier(_hex_centres(c), seed + 77, 1.0) / T

    def advance(v, u, b, alpha, scale):
        de = d * scale
        f = 18.0 * MU_F * DT / (RHO_P * de * de) * alpha
        du = u - v
        vn = torch.where(b, -v, v + _drag(c, du, f, de) * du)
        dep = RHO_P / RHO_F * math.pi * de ** 3 / 6.0 * torch.where(b, torch.zeros_like(v), v - vn)
        return vn, dep

    kept = []
    for n in range(T):
        cell = geo.cell(x)
        u = U[cell].t() * fluid_factor(n)
        none = torch.zeros_like(x, dtype=torch.bool)
        vn, _ = advance(v, u, none, one, one)
        b = geo.wall(x + vn * DT)
        vn, dep = advance(v, u, b, one, one)
        S.index_add_(0, cell, dep.t())
        kept.append((v, cell.int(), b))
        x, v = torch.where(b, x, x + vn * DT), vn
    av = torch.zeros_like(v)
    da = ds = 0.0
    for n in reversed(range(T)):
        v0, cell, b = kept.pop()
        u = U[cell.long()].t() * fluid_factor(n)
        w = [v0.clone().requires_grad_(), one.clone().requires_grad_(), one.clone().requires_grad_()]
        vn, dep = advance(w[0], u, b, w[1], w[2])
        av, ga, gs = torch.autograd.grad((vn * av).sum() + (dep * G[cell.long()].t()).sum(), w)
        da, ds = da + float(ga), ds + float(gs)
    return {"mean": S / T, "dalpha": da, "dscale": ds, "dv0": av}
