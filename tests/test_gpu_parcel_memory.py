"""GPU test that setting, appending and reading parcels needs no device memory beyond the cloud's
own buffers, through which they can be staged: a cloud of more than one chunk (2^20 parcels) that
was made on the device, read back and set again with hardly any memory left, small clouds without
any allocation; and counts at the edges of the staging (an array of cap floats holds cap / 2
doubles), read back exactly."""
import numpy as np
import pytest

import scaletrack as st
import workload

pytestmark = pytest.mark.gpu


def handle(prec, sort_interval=0):
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=1,
                    sort_interval=sort_interval)
    return st.ParcelTracker(prm, st.mesh_desc(8, 0.0, workload.L_BOX))


def parcels(n, prec, seed):
    xyz, _, d = workload.parcels(n, seed)
    uvw = np.random.default_rng(seed).normal(0.0, 0.1, (3, n))
    P = np.float32 if prec == "fp32" else np.float64
    V = np.float64 if prec == "fp64" else np.float32
    return (xyz.astype(P).astype(np.float64), uvw.astype(V).astype(np.float64),
            d.astype(V).astype(np.float64))


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n,m", [(1, 1), (2, 1), (3, 4), (5, 2), (63, 66), (1001, 500)])
def test_edges_of_the_staging(prec, n, m):
    a, b = parcels(n, prec, 80), parcels(m, prec, 81)
    with handle(prec, sort_interval=2) as h:
        h.set_parcels(*a)
        for g, e in zip(h.get_parcels(), a):
            assert np.array_equal(g, e)
        h.append_parcels(*b)
        for g, p, q in zip(h.get_parcels(), a, b):
            assert np.array_equal(g, np.concatenate([p, q], axis=-1))
        h.set_parcels(*b)
        for g, e in zip(h.get_parcels(), b):
            assert np.array_equal(g, e)


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def load_kernels(prec):
    with handle(prec, sort_interval=5) as h:
        h.init_parcels(100, 3, 1e-5, 3e-5)
        a = h.get_parcels()
        h.set_parcels(*a)
        h.append_parcels(*a)


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n", [700_000, (1 << 20) + 12345])
def test_no_memory_left(prec, n):
    import torch
    load_kernels(prec)
    with handle(prec, sort_interval=5) as h:
        h.init_parcels(n, 3, 1e-5, 3e-5)
        full = [torch.empty(free() - (24 << 20), dtype=torch.uint8, device="cuda")]
        try:
            assert free() < 32 << 20
            a = h.get_parcels()
            h.set_parcels(*a)
            b = h.get_parcels()
        finally:
            full.clear()
            torch.cuda.empty_cache()
        c = h.get_parcels()
    for x, y, z in zip(a, b, c):
        assert np.array_equal(x, y) and np.array_equal(x, z)


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
def test_small_clouds_allocate_nothing(prec):
    load_kernels(prec)
    n = 36_000
    with handle(prec) as h:
        h.init_parcels(n, 3, 1e-5, 3e-5)
        before = free()
        a = h.get_parcels()
        h.set_parcels(*a)
        b = h.get_parcels()
        assert free() == before
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
