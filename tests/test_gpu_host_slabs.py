"""Host morphologies of 2^27 voxels: the pitch of a copy that takes several materials
at once (16 bytes a voxel) is then past the 2^31 - 1 bytes that a 2D copy may have,
so the slabs go up one material at a time.  The device-resident call on the same
morphology gives the expected patterns.

Tolerance: the parity tolerance of tests/test_gpu_parity.py, 1e-4 relative on
pixels above 1e-6 of the peak, and identical NaN masks.
"""
import numpy as np
import pytest

from test_gpu_parity import TOL, native, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", [1, 2])
def test_host_call_equals_device_call(strategy):
    nat = native()
    import torch

    n, materials = 512, 2
    gen = torch.Generator(device="cuda").manual_seed(3)
    d_vox = torch.rand((materials, n, n, n, 4), device="cuda", generator=gen)
    d_vox[1, ..., 3] = 1.0 - d_vox[0, ..., 3]
    opts = nat.Options(nx=n, ny=n, nz=n, num_material=materials, energies=[285.0], start_angle=0.0, end_angle=120.0,
                       increment_angle=60.0, phys_size=5.0, rot_mask=1, strategy=strategy)
    optical = np.array([[[4e-3, 1e-3, 2e-3, 5e-4], [1e-3, 3e-4, 1.5e-3, 4e-4]]], np.float32)
    out = torch.zeros((1, 1, n, n), dtype=torch.float32, device="cuda")
    nat.simulate_device(opts, optical, d_vox.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = out.cpu().numpy().astype(np.float64)
    vox = d_vox.cpu().numpy()
    del d_vox
    torch.cuda.empty_cache()
    got = nat.cuda_main(opts, optical, vox).astype(np.float64)
    nat.release_scratch()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert rel_err(got, want).max() <= TOL
