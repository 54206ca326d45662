"""GPU test of the persistent grid of the per-warp step kernel: as many blocks as the instance
that runs keeps resident."""
import numpy as np
import pytest

import scaletrack as st
import workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("clouds", [1, 3])
def test_several_substeps_fill_the_sms(precision, clouds):
    """Its several-substep instances are compiled for three blocks of 256 threads per SM (or
    as many threads in smaller ones), FP64 too, whose one-substep ones are compiled for two."""
    import torch
    prm = st.params(mu_c=workload.MU_F, rho_c=workload.RHO_F, rho_d=workload.RHO_P,
                    drag_model="schiller_naumann", precision=precision, n_substeps=4,
                    n_clouds=clouds)
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    with st.ParcelTracker(prm, st.mesh_desc(12, 0.0, workload.L_BOX)) as h:
        for c in range(clouds):
            h.set_parcels(*workload.parcels(2000, 5 + c), cloud=c)
        h.set_fluid_velocity(workload.tgv_field(12, dtype=np.float32))
        r = h.autotune(workload.DT, trial_steps=4)
        assert r["grid_blocks"] * r["block_size"] >= 3 * 256 * nsm
