"""GPU test of the deposit in planar flows: with a component of every deposit zero the warp run
reduction adds its sums directly instead of handing them over through shared memory, and warps
of both kinds meet in one launch.  Bit-exact with the CPU oracle in the deterministic modes; the
atomic FP64 source within 1e-12 of the oracle's FP64 sum (at most 130 deposits per cell, so
their reordering costs at most 130 * 2^-53 of the sum of magnitudes)."""
import numpy as np
import pytest

import oracle
import scaletrack as st
import workload

pytestmark = pytest.mark.gpu

N = 12


@pytest.mark.parametrize("kind", ["warp", "ring"])
@pytest.mark.parametrize("prec,deposit", [("mixed", "deterministic"), ("fp32", "deterministic"),
                                          ("fp64", "deterministic"), ("fp64", "atomic")])
@pytest.mark.parametrize("zero", [(0,), (1,), (2,), (0, 2), (0, 1, 2)])
def test_planar_deposits(kind, prec, deposit, zero):
    rng = np.random.default_rng(7)
    runs = [1, 3, 8, 9, 31, 32, 2, 40, 130, 1, 1, 5, 16, 17] * 12
    cells = rng.permutation(N ** 3)[:len(runs)]
    cell = np.repeat(cells, runs)
    n = cell.size
    ijk = np.stack([cell % N, (cell // N) % N, cell // (N * N)])
    xyz = (ijk + 0.25 + 0.5 * rng.random((3, n))) * (workload.L_BOX / N)
    uvw = rng.normal(0.0, 0.3, (3, n)).astype(np.float32).astype(np.float64)
    U = rng.normal(0.0, 0.5, (N ** 3, 3)).astype(np.float32)
    for k in zero:
        uvw[k, :2 * n // 3] = 0.0        # the last third has all three components
        U[np.unique(cell[:2 * n // 3]), k] = 0.0
    d = np.full(n, 20e-6, dtype=np.float32).astype(np.float64)
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=1,
                    deposit=deposit)
    with st.ParcelTracker(prm, st.mesh_desc(N, 0.0, workload.L_BOX)) as t:
        t.set_step_kernel(kind)
        t.set_parcels(xyz, uvw, d)
        t.set_fluid_velocity(U)
        t.step(workload.DT)
        t.synchronize()
        gx, gu, _ = t.get_parcels()
        gs = t.get_source()
    cfg = oracle.make_cfg(N, 0.0, workload.L_BOX, workload.MU_F, workload.RHO_F, workload.RHO_P,
                          drag="sn_explicit", precision=prec, n_substeps=1,
                          quant_limbs=2 if prec == "fp64" else 1)
    r = oracle.run(cfg, xyz, uvw, d, U.astype(np.float64), 1, workload.DT)
    assert r["status"] == 0
    assert np.array_equal(gx, r["xyz"])
    assert np.array_equal(gu, r["uvw"])
    if deposit == "deterministic":
        assert np.array_equal(gs, r["src_quant"])
    else:
        assert np.abs(gs - r["src_seq"]).max() <= 1e-12 * np.abs(r["src_seq"]).max()
