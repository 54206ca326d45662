"""GPU test of the relocation shortcuts (a parcel well inside its cell, or well inside the mesh,
is not relocated): parcels on both sides of the limits of each shortcut, against the CPU oracle,
which relocates every parcel in every substep.  Meshes of one to three cells per axis (no inner
cells), of many, and far from the origin (the positions' rounding rules the shortcuts out);
parcels on faces, within 2^-10 of a cell of them, and a few ulp to either side; velocities from
rest to several cells per step, so that parcels bounce and cross; one, ten and 3000 substeps (the
cell coordinate is not followed that long).  Bit-exact in every precision, so also where a
shortcut's bound is not needed."""
import numpy as np
import pytest

import oracle
import scaletrack as st
import workload

pytestmark = pytest.mark.gpu


def parcels(n, rng, npcl, origin, L):
    h = L / n
    ijk = rng.integers(0, n, (3, npcl))
    off = rng.random((3, npcl))
    kind = rng.integers(0, 4, (3, npcl))
    off = np.where(kind == 1, 0.0, off)                                      # on a face
    off = np.where(kind == 2, 2.0 ** -10 * (1 + 0.1 * rng.standard_normal((3, npcl))), off)
    off = np.where(kind == 3, 1 - 2.0 ** -10 * (1 + 0.1 * rng.standard_normal((3, npcl))), off)
    x = origin + (ijk + off) * h
    ulp = rng.integers(-2, 3, (3, npcl))
    x = np.where(kind == 1, np.nextafter(x, np.inf * np.sign(ulp + 0.5)), x)
    lo, hi = origin + 1e-6 * h, origin + L - 1e-4 * h
    x = np.clip(x, lo, hi)
    speed = 10.0 ** rng.uniform(-2, 0.7, npcl) * h / workload.DT             # cells per step
    v = rng.standard_normal((3, npcl)) * speed
    v[:, : npcl // 10] = 0.0
    return x, v.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n,nsub,origin,drag", [
    (1, 1, 0.0, "sn_explicit"), (2, 10, 0.0, "sn_explicit"), (3, 1, 0.0, "sn_explicit"),
    (3, 10, 0.0, "stokes_implicit"), (40, 1, 0.0, "sn_explicit"), (40, 10, -0.03, "sn_explicit"),
    (40, 10, -0.03, "stokes_implicit"), (16, 1, 1000.0, "sn_explicit"),
    (16, 10, 1000.0, "sn_explicit"), (12, 3000, 0.0, "stokes_implicit")])
def test_relocation(prec, n, nsub, origin, drag):
    npcl = 300 if nsub > 100 else 20000
    L = workload.L_BOX * (100.0 if origin > 1 else 1.0)
    rng = np.random.default_rng(100 + n + nsub)
    xyz, uvw = parcels(n, rng, npcl, origin, L)
    if prec == "fp32":
        xyz = np.clip(xyz.astype(np.float32), np.nextafter(np.float32(origin), np.float32(1e9)),
                      np.nextafter(np.float32(origin + L), np.float32(-1e9))).astype(np.float64)
    d = (30e-6 * np.exp(0.2 * rng.standard_normal(npcl))).astype(np.float32).astype(np.float64)
    U = rng.standard_normal((n ** 3, 3)).astype(np.float64 if prec == "fp64" else np.float32)
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model=drag, precision=prec, n_substeps=nsub)
    cfg = oracle.make_cfg(n, origin, origin + L, workload.MU_F, workload.RHO_F, workload.RHO_P,
                          drag=drag, precision=prec, n_substeps=nsub,
                          quant_limbs=2 if prec == "fp64" else 1)
    r = oracle.run(cfg, xyz, uvw, d, U.astype(np.float64), 3, workload.DT, nthreads=8)
    for kernel in ("warp", "ring"):
        with st.ParcelTracker(prm, st.mesh_desc(n, origin, origin + L)) as h:
            h.set_step_kernel(kernel)
            h.set_parcels(xyz, uvw, d)
            h.set_fluid_velocity(U)
            for _ in range(3):
                h.step(workload.DT)
            x, u, _ = h.get_parcels(check=r["status"] == 0)
            s = h.get_source(check=False)
        assert np.array_equal(x, r["xyz"])
        assert np.array_equal(u, r["uvw"])
        assert np.array_equal(s, r["src_quant"])
