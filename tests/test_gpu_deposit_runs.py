"""GPU test of the deposit's warp run reduction: runs of equal cells of every length around the
edges of its chunks (8 lanes), of a warp (32) and of a warp tile, in every deposit mode.  One
cell per run in order of the parcels, so the run lengths are what the kernel meets; with
`heavy` some parcels are 2^9 times heavier, which takes their warps past the 32-bit path.
Positions, velocities and the fixed-point source are bit-exact with the CPU oracle (the
integers do not depend on how runs are cut), the atomic FP64 source within 1e-12 of the
oracle's FP64 sum: every cell sums at most 130 deposits, so the reordering costs at most
130 * 2^-53 of the sum of magnitudes, below 1.5e-14."""
import numpy as np
import pytest

import oracle
import scaletrack as st
import workload

pytestmark = pytest.mark.gpu

N = 16
LENGTHS = [1, 2, 7, 8, 9, 15, 16, 17, 1, 1, 31, 32, 33, 3, 64, 65, 5, 130]


@pytest.mark.parametrize("kind", ["warp", "ring"])
@pytest.mark.parametrize("prec,deposit", [("mixed", "deterministic"), ("fp32", "deterministic"),
                                          ("fp64", "deterministic"), ("fp64", "atomic"),
                                          ("mixed", "atomic")])
@pytest.mark.parametrize("heavy", [False, True])
def test_runs_of_every_length(kind, prec, deposit, heavy):
    rng = np.random.default_rng(31)
    runs = LENGTHS * 12
    cells = rng.permutation(N ** 3)[:len(runs)]
    cell = np.repeat(cells, runs)
    n = cell.size
    h = workload.L_BOX / N
    ijk = np.stack([cell % N, (cell // N) % N, cell // (N * N)])
    xyz = (ijk + 0.25 + 0.5 * rng.random((3, n))) * h
    uvw = rng.normal(0.0, 0.3, (3, n)).astype(np.float32).astype(np.float64)
    d = np.full(n, 20e-6)
    if heavy:
        d[rng.random(n) < 0.02] *= 8.0
    d = d.astype(np.float32).astype(np.float64)
    U = workload.tgv_field(N, dtype=np.float64 if prec == "fp64" else np.float32)
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=1,
                    deposit=deposit)
    with st.ParcelTracker(prm, st.mesh_desc(N, 0.0, workload.L_BOX)) as t:
        t.set_step_kernel(kind)
        t.set_parcels(xyz, uvw, d)
        t.set_fluid_velocity(U)
        for _ in range(2):
            t.step(workload.DT)
        t.synchronize()
        gx, gu, _ = t.get_parcels()
        gs = t.get_source()
    cfg = oracle.make_cfg(N, 0.0, workload.L_BOX, workload.MU_F, workload.RHO_F, workload.RHO_P,
                          drag="sn_explicit", precision=prec, n_substeps=1,
                          quant_limbs=2 if prec == "fp64" else 1)
    r = oracle.run(cfg, xyz, uvw, d, U.astype(np.float64), 2, workload.DT)
    assert r["status"] == 0
    assert np.array_equal(gx, r["xyz"])
    assert np.array_equal(gu, r["uvw"])
    if deposit == "deterministic":
        assert np.array_equal(gs, r["src_quant"])
    else:
        ref = r["src_seq"]
        assert np.abs(gs - ref).max() <= 1e-12 * np.abs(ref).max()
