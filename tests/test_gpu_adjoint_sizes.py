"""GPU test of the pull-back at the sizes where its blocks change: parcel counts around one
block of 256 and around more blocks than stay resident, segments that do not divide the steps,
checkpoints every step and never, fast parcels that bounce and change cells on most steps, and
drag parameters of one (their divisions are left out) and not of one.  Mean source and velocity
cotangents bit for bit against the CPU adjoint, parameter gradients to FP64 summation order
(at most 2e5 terms of one sign or another: 1e-10 of the sum of magnitudes, taken from dv0's
scale, is far above n * 2^-53)."""
import numpy as np
import pytest

import oracle
import scaletrack as st
import workload

pytestmark = pytest.mark.gpu

N = 6


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("npcl,T,C,alpha,s", [(1, 5, 5, 1.0, 1.0), (255, 7, 3, 1.0, 1.0),
                                              (257, 6, 1, 1.3, 0.9), (512, 9, 100, 1.0, 0.9),
                                              (148 * 4 * 256 + 300, 4, 3, 1.3, 1.0)])
def test_pullback_sizes(prec, npcl, T, C, alpha, s):
    xyz, _, d = workload.parcels(npcl, 80)
    uvw = np.random.default_rng(81).normal(0.0, 30.0, (3, npcl)).astype(np.float32).astype(float)
    U = workload.tgv_field(N, U0=2.0, dtype=np.float64 if prec == "fp64" else np.float32)
    fs = np.array([workload.fluid_scale(k) for k in range(T)])
    cot = np.random.default_rng(82).standard_normal((N ** 3, 3)) * 1e-9
    limbs = 2 if prec == "fp64" else 1
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=1,
                    drag_multiplier=alpha, diameter_scale=s, sort_interval=3)
    with st.ParcelTracker(prm, st.mesh_desc(N, 0.0, workload.L_BOX)) as h:
        h.set_parcels(xyz, uvw, d)
        h.set_fluid_velocity(U)
        S = h.mean_source_forward(T, C, workload.DT, fs)
        da, ds, dv0 = h.mean_source_pullback(cot, T, C, workload.DT, fs)
        da2, ds2, none = h.mean_source_pullback(cot, T, C, workload.DT, fs, want_v0=False)
    assert none is None and (da, ds) == (da2, ds2)
    cfg = oracle.make_cfg(N, 0.0, workload.L_BOX, workload.MU_F, workload.RHO_F, workload.RHO_P,
                          drag="sn_explicit", precision=prec, n_substeps=1,
                          drag_multiplier=alpha, diameter_scale=s)
    r = oracle.adjoint(cfg, xyz, uvw, d, U, T, workload.DT, fscale=fs, cotangent=cot,
                       mean_limbs=limbs)
    assert r["status"] == 0
    assert np.array_equal(S, r["mean_src"])
    assert np.array_equal(dv0, r["dv0"])
    assert abs(da - r["dalpha"]) <= 1e-10 * abs(r["dalpha"])
    assert abs(ds - r["dscale"]) <= 1e-10 * abs(r["dscale"])
