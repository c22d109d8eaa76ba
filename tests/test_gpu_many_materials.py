"""FIELDS requests with more materials than the Ewald kernel walks at compile time,
up to the 32 that the options allow (every term formed; the coefficients of the
packed volumes staged in shared memory), alone and as a request group.

Tolerance: the parity tolerance of tests/test_gpu_parity.py, 1e-4 relative on
pixels above 1e-6 of the peak, and identical NaN masks.
"""
import numpy as np
import pytest

import cases
import oracle
from test_gpu_parity import TOL, native, options_for, rel_err

pytestmark = pytest.mark.gpu

FRAMES = {"lab": {}, "tilted": dict(case_type=1, kvecs=[[0.05, 0.02, 1.0]]), "material": dict(frame=cases.MATERIAL)}


def _case(materials, **over):
    return cases.Case("many", 26, 22, 6, materials, [282.0, 284.0, 285.0, 286.0, 289.0], seed=materials,
                      geometry="blobs", angles=(0.0, 150.0, 50.0), rot_mask=1, **over)


@pytest.mark.parametrize("frame", FRAMES)
@pytest.mark.parametrize("materials", [9, 18, 19, 32])
def test_matches_oracle(materials, frame):
    case = _case(materials, **FRAMES[frame])
    optical, vox = cases.optical_constants(case), cases.voxels(case)
    got = native().cuda_main(options_for(case, strategy=2), optical, vox).astype(np.float64)
    want = oracle.run_case(case)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert rel_err(got, want).max() <= TOL


@pytest.mark.parametrize("materials", [19, 32])
def test_group_matches_alone(materials):
    nat = native()
    import torch

    from cyrsoxs_gb300 import serving

    case = _case(materials)
    optical, vox = cases.optical_constants(case), np.ascontiguousarray(cases.voxels(case), np.float32)
    opts = options_for(case, strategy=2)
    want = nat.cuda_main(opts, optical, vox).astype(np.float64)
    d_vox = torch.from_numpy(vox).cuda()
    outs = [torch.zeros(want.shape, dtype=torch.float32, device="cuda") for _ in range(6)]
    torch.cuda.synchronize()
    with serving.Server(slots=1, groups=True) as srv:
        ids = [srv.submit(opts, optical, d_vox.data_ptr(), o.data_ptr(), device=True) for o in outs]
        for i in ids:
            srv.wait(i)
        assert srv.stats()["grouped_requests"] > 0
    for o in outs:
        got = o.cpu().numpy().astype(np.float64)
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert rel_err(got, want).max() <= TOL
