"""GPU test of the small-cloud step: the per-warp kernel with the source conversion launched
behind it in stream order (programmatic dependent launch), which the library takes by itself for
small clouds, against the ring kernel with the conversion on the second stream and against the
CPU oracle.  Several steps run without a host synchronisation, each with another carrier field
copied in between, and the parcels are replaced once so that cells with a source lose it (the
conversion clears only what was added to).  Everything is bit-exact: both paths run the same
parcel arithmetic and integer sums."""
import numpy as np
import pytest

import oracle
import scaletrack as st
import workload

pytestmark = pytest.mark.gpu

N = 10
STEPS = 5


def fields(prec):
    dt = np.float64 if prec == "fp64" else np.float32
    return [(workload.tgv_field(N, U0=1.0 + 0.5 * k) + 0.1 * k).astype(dt) for k in range(STEPS)]


def run(prec, nsub, n, kernel, overlap, stream0, seed):
    import torch
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=nsub)
    Us = [torch.tensor(u, device="cuda") for u in fields(prec)]
    torch.cuda.synchronize()
    out = []
    with st.ParcelTracker(prm, st.mesh_desc(N, 0.0, workload.L_BOX)) as h:
        if stream0:
            st.lib().st_set_stream(h.handle, None)
        if kernel:
            h.set_step_kernel(kernel)
        h.set_finalize_overlap(overlap)
        for rep in range(2):
            xyz, uvw, d = workload.parcels(n, seed + rep)
            h.set_parcels(xyz, uvw, d)
            for k in range(STEPS):
                h.set_fluid_velocity_device(Us[k].data_ptr(), Us[k].element_size())
                h.step(workload.DT, workload.fluid_scale(k))
            s = h.get_source()
            x, u, _ = h.get_parcels()
            out.append((x, u, h.get_cells(), s))
    return out


@pytest.mark.parametrize("n", [1, 33, 256, 20011])
@pytest.mark.parametrize("prec,nsub", [("fp32", 1), ("mixed", 1), ("mixed", 3), ("fp64", 1)])
def test_small_cloud_paths_agree(prec, nsub, n):
    a = run(prec, nsub, n, None, True, False, 50)
    for other in (run(prec, nsub, n, "ring", True, False, 50),
                  run(prec, nsub, n, None, True, True, 50),
                  run(prec, nsub, n, None, False, False, 50)):
        for p, q in zip(a, other):
            for x, y in zip(p, q):
                assert np.array_equal(x, y)
    # the last carrier field alone against the oracle, from rest
    xyz, uvw, d = workload.parcels(n, 50)
    U = fields(prec)[0]
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=nsub)
    with st.ParcelTracker(prm, st.mesh_desc(N, 0.0, workload.L_BOX)) as h:
        h.set_parcels(xyz, uvw, d)
        h.set_fluid_velocity(U)
        for _ in range(3):
            h.step(workload.DT)
        g = (*h.get_parcels()[:2], h.get_cells(), h.get_source())
    cfg = oracle.make_cfg(N, 0.0, workload.L_BOX, workload.MU_F, workload.RHO_F, workload.RHO_P,
                          drag="sn_explicit", precision=prec, n_substeps=nsub,
                          quant_limbs=2 if prec == "fp64" else 1)
    r = oracle.run(cfg, xyz, uvw, d, U.astype(np.float64), 3, workload.DT)
    assert r["status"] == 0
    for x, y in zip(g, (r["xyz"], r["uvw"], r["cells"], r["src_quant"])):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("npcl", [0, 1, 33, 3001])
def test_noalloc_calls_in_a_row(npcl):
    """The allocation-free step uses two control sets in turn, each reset by the call before:
    five calls in a row, one of them with a parcel outside the mesh (its error is its own) and
    on alternating streams, each give the source of a fresh handle that steps the same parcels
    (the scale comes from each call's own largest deposit, as a fresh handle's first step)."""
    import ctypes
    import torch
    n = 9
    xyz, uvw, d = workload.parcels(max(npcl, 1), 90)
    xyz, uvw, d = xyz[:, :npcl], uvw[:, :npcl], d[:npcl]
    U = workload.tgv_field(n, dtype=np.float32)
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision="mixed", n_substeps=1)
    mesh = st.mesh_desc(n, 0.0, workload.L_BOX)
    dev = torch.device("cuda", 0)
    X = [torch.tensor(a, dtype=torch.float64, device=dev) for a in xyz]
    V = [torch.tensor(a, dtype=torch.float32, device=dev) for a in uvw]
    D = torch.tensor(d, dtype=torch.float32, device=dev)
    Ud = torch.tensor(U, device=dev)
    S = torch.full((n ** 3, 3), float("nan"), dtype=torch.float64, device=dev)
    streams = [torch.cuda.default_stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()

    def call(k):
        p = ctypes.c_void_p
        return st.lib().st_step_noalloc(
            ctypes.byref(prm), ctypes.byref(mesh), npcl, *[p(t.data_ptr() or None) for t in X],
            *[p(t.data_ptr() or None) for t in V], p(D.data_ptr() or None), p(Ud.data_ptr()),
            p(S.data_ptr()), workload.DT, 1.0, p(streams[k % 2].cuda_stream))

    for k in range(5):
        if npcl > 1 and k == 2:      # a call that reports a lost parcel
            keep = X[0][0].item()
            X[0][0] = 2.5 * workload.L_BOX
            torch.cuda.synchronize()
            assert call(k) == st.ST_ERR_PARCEL_OUTSIDE
            X[0][0] = keep
            torch.cuda.synchronize()
            continue
        ref = np.zeros((n ** 3, 3))
        if npcl:
            x = np.stack([t.cpu().numpy() for t in X])
            v = np.stack([t.cpu().numpy().astype(np.float64) for t in V])
            with st.ParcelTracker(prm, mesh) as h:
                h.set_parcels(x, v, d)
                h.set_fluid_velocity(U)
                h.step(workload.DT)
                ref = h.get_source()
                px, pv, _ = h.get_parcels()
        assert call(k) == st.ST_OK, st.last_error()
        assert np.array_equal(S.cpu().numpy(), ref)
        if npcl:
            assert np.array_equal(np.stack([t.cpu().numpy() for t in X]), px)
            assert np.array_equal(np.stack([t.cpu().numpy() for t in V]).astype(np.float64), pv)


class _DeviceArray:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False),
                                             version=2)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [3, 5, 11])
def test_sources_empty_where_parcels_left(prec, n):
    """The conversion clears an accumulator only where something was added, and writes the whole
    source also over what its holder wrote there: three clouds (one empty, one in a corner, one
    everywhere) whose parcels are replaced twice, with component counts that leave ragged groups
    of four.  Each source, in 8 and 4 bytes, equals that of a handle that never held others."""
    import torch
    U = workload.tgv_field(n, U0=2.0, dtype=np.float64 if prec == "fp64" else np.float32)
    mesh = st.mesh_desc(n, 0.0, workload.L_BOX)

    def prm(nc):
        return st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                         drag_model="schiller_naumann", precision=prec, n_substeps=1, n_clouds=nc)

    def clouds(rep):
        out = []
        for c, npcl in enumerate((0, 40, 700)):
            xyz, uvw, d = workload.parcels(npcl, 7 * rep + c)
            if c == 1:
                xyz = xyz / n if rep % 2 == 0 else workload.L_BOX * (1 - 1e-6) - xyz / n
            out.append((xyz, uvw, d))
        return out

    with st.ParcelTracker(prm(3), mesh) as h:
        h.set_fluid_velocity(U)
        for rep in range(3):
            for c, p in enumerate(clouds(rep)):
                h.set_parcels(*p, cloud=c)
            h.step(workload.DT)
            h.synchronize()
            for c in range(3):
                src = _DeviceArray(h.source_device_ptr(c), 3 * n**3)
                torch.as_tensor(src, device="cuda").fill_(1.5)
            torch.cuda.synchronize()
            h.step(workload.DT)
            for c, p in enumerate(clouds(rep)):
                with st.ParcelTracker(prm(1), mesh) as f:
                    f.set_fluid_velocity(U)
                    f.set_parcels(*p)
                    for _ in range(2):
                        f.step(workload.DT)
                    ref = f.get_source()
                got = h.get_source(cloud=c)
                assert np.array_equal(got, ref)
                assert np.array_equal(h.get_source(cloud=c, dtype=np.float32), ref.astype(np.float32))
                assert (np.abs(ref).max() > 0) == (c > 0)
