"""An FP64 request that asks for the field spectra but has no room for their volumes
runs with per-energy spectra instead of failing: 32 materials take 112 volumes of
16 bytes a voxel, the per-energy spectra five.  The rest of the device's memory is
taken up meanwhile.
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import native, options_for

pytestmark = pytest.mark.gpu


def test_fields_that_do_not_fit():
    nat = native()
    import torch

    case = cases.Case("memory", 96, 96, 96, 32, [283.0], seed=9, angles=(0.0, 120.0, 60.0), rot_mask=1)
    optical, vox = cases.optical_constants(case), np.ascontiguousarray(cases.voxels(case), np.float32)
    d_vox = torch.from_numpy(vox).cuda()
    out = torch.zeros((1, 1, 96, 96), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def run(strategy):
        nat.simulate_device_fp64(options_for(case, strategy=strategy), optical, d_vox.data_ptr(), False, out.data_ptr(),
                                 stream)
        torch.cuda.synchronize()
        return out.cpu().numpy()

    want = run(1).copy()
    nat.release_scratch()
    torch.cuda.empty_cache()
    volumes = 112 * 96**3 * 16
    free, _ = torch.cuda.mem_get_info()
    rest = torch.empty(free - volumes // 2, dtype=torch.uint8, device="cuda")
    try:
        got = run(2)
    finally:
        del rest
        torch.cuda.empty_cache()
        nat.release_scratch()
    assert np.array_equal(got, want, equal_nan=True)
