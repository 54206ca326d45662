"""GPU test of the device memory of the adjoint's records: with a few parcels it follows their
number, however long the checkpoint interval; where the records of every resident block do not
fit, fewer blocks run.  Gradients are the same bits as with short intervals and memory to spare
(every parcel's steps are summed in one order)."""
import numpy as np
import pytest

import scaletrack as st
import workload

pytestmark = pytest.mark.gpu

N = 8


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def handle(n, prec):
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=prec, n_substeps=1)
    h = st.ParcelTracker(prm, st.mesh_desc(N, 0.0, workload.L_BOX))
    xyz, uvw, d = workload.parcels(n, 90)
    h.set_parcels(xyz, uvw, d)
    h.set_fluid_velocity(workload.tgv_field(N, dtype=np.float64 if prec == "fp64" else np.float32))
    return h


def gradients(h, cot, T, C):
    S = h.mean_source_forward(T, C, workload.DT)
    return (S,) + tuple(h.mean_source_pullback(cot, T, C, workload.DT))


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [1, 33, 255])
def test_few_parcels_long_interval(prec, n):
    T = 20_000
    cot = np.random.default_rng(91).normal(0.0, 1.0, (N ** 3, 3))
    with handle(n, prec) as h:
        ref = gradients(h, cot, 200, 7)
        one = gradients(h, cot, 200, 200)
        assert same(ref, one)
        before = free()
        long = gradients(h, cot, T, T)
        # records of 4 velocities, a cell and a flag per parcel and step, n rounded up to 32
        need = T * ((n + 31) // 32 * 32) * ((32 if prec == "fp64" else 16) + 5)
        assert before - free() <= need + (4 << 20)
        assert same(long, gradients(h, cot, T, 500))


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_fewer_blocks_where_the_records_do_not_fit(prec):
    import torch
    T, C, n = 300, 300, 40_000
    cot = np.random.default_rng(92).normal(0.0, 1.0, (N ** 3, 3))
    with handle(n, prec) as h:
        ref = gradients(h, cot, T, C)          # 252 MB of records in mixed precision
    with handle(n, prec) as h:
        gradients(h, cot, 2, 1)
        full = [torch.empty(free() - (96 << 20), dtype=torch.uint8, device="cuda")]
        try:
            assert same(gradients(h, cot, T, C), ref)
        finally:
            full.clear()
            torch.cuda.empty_cache()
