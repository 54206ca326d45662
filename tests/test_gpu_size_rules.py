"""GPU test of the rules by size on both sides of their lines: where the accumulators of many clouds
are cleared (by the conversion up to 24 MB and above 96 MB, by a memset between), and one handle
whose cloud is replaced and grows across the lines between programmatic launches, the ring and the
conversion on the second stream.  Bit-identical to handles of one cloud, and to fresh handles with
the per-warp kernel and every conversion in stream order."""
import numpy as np
import pytest

import scaletrack as st
import workload

pytestmark = pytest.mark.gpu


def handle(prec, mesh, clouds=1, **kw):
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=1, n_clouds=clouds,
                    **kw)
    return st.ParcelTracker(prm, st.mesh_desc(mesh, 0.0, workload.L_BOX))


def steps(h, k):
    for i in range(k):
        h.step(workload.DT, workload.fluid_scale(i, workload.DT, True))


@pytest.mark.parametrize("prec,clouds", [("mixed", 3), ("mixed", 5), ("mixed", 15), ("mixed", 16),
                                         ("fp64", 2), ("fp64", 7), ("fp64", 8)])
def test_clearing_of_many_clouds(prec, clouds):
    """64^3 cells: 6.3 MB of accumulators a cloud, twice that in FP64."""
    n = 64
    U = workload.tgv_field(n, dtype=np.float64 if prec == "fp64" else np.float32)
    sets = [[workload.parcels(300 + 17 * c, 200 + 20 * r + c) for c in range(clouds)]
            for r in range(2)]
    out = [[] for _ in range(clouds)]
    with handle(prec, n, clouds) as h:
        h.set_fluid_velocity(U)
        for r in range(2):
            for c in range(clouds):
                h.set_parcels(*sets[r][c], cloud=c)
            for _ in range(2):
                steps(h, 1)
                for c in range(clouds):
                    out[c].append(h.get_source(c))
    for c in range(clouds):
        with handle(prec, n) as h:
            h.set_finalize_overlap(0)
            h.set_fluid_velocity(U)
            k = 0
            for r in range(2):
                h.set_parcels(*sets[r][c])
                for _ in range(2):
                    steps(h, 1)
                    S = h.get_source()
                    assert np.abs(S).max() > 0
                    assert np.array_equal(out[c][k], S), (c, k)
                    k += 1


@pytest.mark.parametrize("prec,mesh,counts", [
    ("mixed", 20, [2000, 600_000, 1_600_000, 3000]),      # ring from 1.5e6 on, 5e5 launches
    ("mixed", 72, [40_000, 60_000, 30_000]),              # accumulators above 8 MB: from 5e4 on
    ("mixed", 60, [200_000, 260_000, 100_000]),           # meshes above 2e5 cells: 2.5e5
    ("fp64", 20, [440_000, 460_000, 20_000]),             # FP64: 4.5e5
    ("fp32", 20, [1_400_000, 1_600_000, 10]),
])
def test_one_handle_across_the_rules(prec, mesh, counts):
    U = workload.tgv_field(mesh, dtype=np.float64 if prec == "fp64" else np.float32)
    sets = [workload.parcels(n, 300 + k) for k, n in enumerate(counts)]

    def run(h, p):
        h.set_parcels(*p)
        steps(h, 3)
        return h.get_source(), h.get_parcels()[0]

    with handle(prec, mesh) as h:
        h.set_fluid_velocity(U)
        got = [run(h, p) for p in sets]
        # the last cloud grows over the second line
        m = counts[1] - counts[-1] + 5
        h.append_parcels(*[a[..., :m] for a in sets[1]])
        steps(h, 3)
        grown = h.get_source()
    for p, (S, x) in zip(sets, got):
        with handle(prec, mesh) as h:
            h.set_step_kernel("warp")
            h.set_finalize_overlap(0)
            h.set_fluid_velocity(U)
            S0, x0 = run(h, p)
            assert np.abs(S0).max() > 0
            assert np.array_equal(S, S0) and np.array_equal(x, x0)
            last = h if p is sets[-1] else None
            if last:
                h.append_parcels(*[a[..., :m] for a in sets[1]])
                steps(h, 3)
                assert np.array_equal(grown, h.get_source())


def test_atomic_deposit_across_the_rules():
    """On a mesh whose accumulators would be above 8 MB; the sums within 1e-12 of the per-warp
    kernel's (a cell's few deposits in another order: some 2^-53 of the sum of magnitudes)."""
    U = workload.tgv_field(72, dtype=np.float64)
    for n in (60_000, 440_000, 460_000):
        p = workload.parcels(n, 310)
        out = []
        for kind in (None, "warp"):
            with handle("fp64", 72, deposit="atomic") as h:
                if kind:
                    h.set_step_kernel(kind)
                h.set_fluid_velocity(U)
                h.set_parcels(*p)
                steps(h, 3)
                out.append((h.get_source(), h.get_parcels()[0]))
        assert np.array_equal(out[0][1], out[1][1])
        assert np.abs(out[0][0] - out[1][0]).max() <= 1e-12 * np.abs(out[1][0]).max()
