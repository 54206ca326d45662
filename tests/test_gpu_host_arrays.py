"""GPU test of the copies between device memory and the caller's host arrays: parcel counts and
mesh sizes on both sides of the sizes where the copies go through the staging buffers (2 MB),
where their pieces change (16 MB) and where the parcels take more than one chunk (2^20), pageable
and pinned arrays, and two host threads at once.  Parcels come back as they were set (rounded to
the precision's types), the source in 4 and 8 bytes, and the cells as the oracle locates them."""
import threading

import numpy as np
import pytest

import scaletrack as st
import workload

pytestmark = pytest.mark.gpu


def handle(prec, n, **kw):
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=1, **kw)
    return st.ParcelTracker(prm, st.mesh_desc(n, 0.0, workload.L_BOX))


def roundtrip(prec, npcl, sort_interval=4, seed=60):
    xyz, uvw, d = workload.parcels(npcl, seed)
    uvw = np.random.default_rng(seed).normal(0.0, 0.1, (3, npcl))
    with handle(prec, 8, sort_interval=sort_interval) as h:
        h.set_parcels(xyz, uvw, d)
        x, u, dd = h.get_parcels()
        cells, order = h.get_cells(), h.get_order()
    P = np.float32 if prec == "fp32" else np.float64
    V = np.float64 if prec == "fp64" else np.float32
    assert np.array_equal(x, xyz.astype(P).astype(np.float64))
    assert np.array_equal(u, uvw.astype(V).astype(np.float64))
    assert np.array_equal(dd, d.astype(V).astype(np.float64))
    assert np.array_equal(np.sort(order), np.arange(npcl))
    L = np.float64(workload.L_BOX)
    rd = P(1.0 / (L / 8))
    i = np.floor(xyz.astype(P) * rd).astype(np.int64)
    assert np.array_equal(cells, (i[2] * 8 + i[1]) * 8 + i[0])


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("npcl", [1, 37000, 299_600, (1 << 20) - 1, (1 << 20) + 1])
def test_parcels_come_back(prec, npcl):
    roundtrip(prec, npcl)


@pytest.mark.parametrize("n", [10, 44, 45, 89, 96])
def test_fields_pageable_and_pinned(n):
    """2 MB lie between 44^3 and 45^3 doubles [n][3], 16 MB between 88^3 and 89^3."""
    import torch
    xyz, uvw, d = workload.parcels(5000, 61)
    U = workload.tgv_field(n, dtype=np.float64)
    Up = torch.empty(U.shape, dtype=torch.float64, pin_memory=True).numpy()
    Up[:] = U
    out = []
    for u in (U, Up, U.astype(np.float32)):
        with handle("mixed", n) as h:
            h.set_parcels(xyz, uvw, d)
            h.set_fluid_velocity(u)
            h.step(workload.DT)
            s8, s4 = h.get_source(), h.get_source(dtype=np.float32)
            S = torch.empty(U.shape, dtype=torch.float64, pin_memory=True).numpy()
            assert st.lib().st_get_source(h.handle, 0, S.ctypes.data, 8) == 0
            assert np.array_equal(S, s8) and np.array_equal(s4, s8.astype(np.float32))
            out.append(s8)
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    assert np.abs(out[0]).max() > 0


def test_two_host_threads():
    errs = []

    def work(seed):
        try:
            for k in range(3):
                roundtrip("mixed", 400_000, seed=seed + k)
        except Exception as e:  # noqa: BLE001
            errs.append(e)

    ts = [threading.Thread(target=work, args=(70 + 10 * t,)) for t in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errs, errs
