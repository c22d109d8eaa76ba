"""Served device buffers that the kernels cannot address in place, a morphology off its
16 bytes or a projection off its 4, go through the slot's staging buffers, with graphs
and groups as without.  Each request equals the same request on aligned buffers.

Tolerance: the parity tolerance of tests/test_gpu_parity.py, 1e-4 relative on pixels
above 1e-6 of the peak, and identical NaN masks.
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import TOL, native, options_for, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", [1, 2])
@pytest.mark.parametrize("graphs,groups", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("vox_off,out_off", [(4, 0), (0, 2), (8, 1)])
def test_unaligned_buffers(strategy, graphs, groups, vox_off, out_off):
    nat = native()
    import torch

    from cyrsoxs_gb300 import serving

    case = cases.Case("alignment", 40, 36, 8, 2, [284.0, 286.0], seed=3, geometry="blobs", angles=(0.0, 120.0, 60.0),
                      rot_mask=1)
    opts, optical = options_for(case, strategy=strategy), cases.optical_constants(case)
    vox = np.ascontiguousarray(cases.voxels(case), np.float32)
    want = nat.cuda_main(opts, optical, vox)
    d_vox = torch.zeros(vox.nbytes + 16, dtype=torch.uint8, device="cuda")
    d_vox[vox_off:vox_off + vox.nbytes] = torch.from_numpy(vox.reshape(-1).view(np.uint8)).cuda()
    outs = [torch.zeros(want.nbytes + 16, dtype=torch.uint8, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    with serving.Server(slots=1, graphs=graphs, groups=groups) as srv:
        ids = [srv.submit(opts, optical, d_vox.data_ptr() + vox_off, o.data_ptr() + out_off, device=True) for o in outs]
        for i in ids:
            srv.wait(i)
    for o in outs:
        got = o[out_off:out_off + want.nbytes].cpu().numpy().view(np.float32).reshape(want.shape).astype(np.float64)
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert rel_err(got, want.astype(np.float64)).max() <= TOL
