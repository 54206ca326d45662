"""GPU test of the tet ring's two instances of the walk (neighbours beside the planes on re-sorted
clouds with FP32 velocities, one neighbour at a time otherwise): parcels, owning tets, walk lengths
and the fixed-point source are bit-identical to the per-warp kernel's, long walks and bounces
included, in every precision, deposit and number of substeps that has an instance."""
import numpy as np
import pytest

import scaletrack as st
import workload

pytestmark = pytest.mark.gpu

L = workload.L_BOX


@pytest.mark.parametrize("sort", [0, 2])
@pytest.mark.parametrize("prec,deposit", [("mixed", "deterministic"), ("mixed", "atomic"),
                                          ("fp64", "deterministic")])
@pytest.mark.parametrize("sub", [1, 3])
def test_ring_walks(sort, prec, deposit, sub):
    n, m = 6, 992 * 3 + 17
    verts, tets, nbr, hex_ijk = workload.kuhn_tet_mesh(n, L, 0.15, 1)
    xyz, _, d = workload.parcels(m, 400, d_median=40e-6)
    uvw = np.random.default_rng(401).normal(0.0, 20.0, (3, m)).astype(np.float32).astype(float)
    U = workload.tgv_at(workload.tet_centroids(verts, tets), U0=3.0)
    U = U if prec == "fp64" else U.astype(np.float32)
    hint = workload.tet_hints(xyz, hex_ijk, n, L)
    out = []
    for kind in ("ring", "warp"):
        prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                        drag_model="schiller_naumann", precision=prec, n_substeps=sub,
                        deposit=deposit, sort_interval=sort)
        with st.ParcelTracker(prm, st.tet_mesh_desc(verts, tets, nbr, 0.0, L)) as h:
            h.set_step_kernel(kind)
            h.set_parcels(xyz, uvw, d, hint=hint)
            h.set_fluid_velocity(U)
            for _ in range(5):
                h.step(1e-3)
            h.synchronize()
            x, v, _ = h.get_parcels()
            out.append((x, v, h.get_cells(), np.array(h.hop_histogram()), h.get_source()))
    for a, b in zip(out[0][:4], out[1][:4]):
        assert np.array_equal(a, b)
    assert out[0][3][2:].sum() > 0
    if deposit == "deterministic":
        assert np.array_equal(out[0][4], out[1][4])
    else:
        assert np.abs(out[0][4] - out[1][4]).max() <= 1e-12 * np.abs(out[1][4]).max()
