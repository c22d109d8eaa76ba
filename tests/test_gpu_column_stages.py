"""Column passes over TMA tiles when every block takes many more tiles than it
has stages, so each stage is stored and loaded again: the exchange inside the
tile (128- and 256-point lines) or beside it (512), and the masked z pass, whose
boxes are stored a lane each.

Tolerances: the transform's 2e-6 of the largest value and the parity tolerance of
tests/test_gpu_parity.py, 1e-4 relative on pixels above 1e-6 of the peak.
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import TOL, _torch, native, options_for, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,count", [((128, 128, 224), 2), ((128, 128, 112), 3), ((256, 256, 96), 2),
                                         ((512, 16, 512), 2), ((8, 512, 1008), 1)])
def test_transform_matches_double(shape, count):
    torch = _torch()
    nz, ny, nx = shape
    gen = torch.Generator(device="cuda").manual_seed(nx)
    a = torch.randn((count,) + shape + (2,), device="cuda", generator=gen)
    ref = torch.fft.fftn(torch.view_as_complex(a.double()), dim=(1, 2, 3))
    native().fft3d_device(a.data_ptr(), nx, ny, nz, count, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    err = (torch.view_as_complex(a).to(torch.complex128) - ref).abs().max() / ref.abs().max()
    assert float(err) < 2e-6, float(err)


@pytest.mark.parametrize("nx,ny,nz", [(128, 96, 256), (144, 80, 128), (96, 48, 512)])
def test_masked_z_pass_matches_per_energy_spectra(nx, ny, nz):
    case = cases.Case("stages", nx, ny, nz, 3, [284.0, 286.0], seed=nz, geometry="blobs", angles=(0.0, 120.0, 60.0),
                      rot_mask=1)
    optical, vox = cases.optical_constants(case), cases.voxels(case)
    nat = native()
    nat.profile_begin()
    got = nat.cuda_main(options_for(case, strategy=2), optical, vox).astype(np.float64)
    launched, _ = nat.profile_end()
    assert "k_zmask" in launched
    want = nat.cuda_main(options_for(case, strategy=1), optical, vox).astype(np.float64)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert rel_err(got, want).max() <= 2 * TOL  # both sides within TOL of the exact result
