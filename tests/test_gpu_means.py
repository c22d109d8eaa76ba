"""The constants taken out of the fields before the transform come from a sample of
the morphology.  They must lie near the means wherever the structure lies, or the
float32 rounding of the transform grows with what is left of them.  A morphology
turned cyclically along an axis has the same intensities, so its error against the
FP64 pipeline must be the same: a grating along y whose pitch is the step of a
sample by rows, and a film with thin layers.  The contrasts are opposite (a
third, absent material without contrast lies between them), so no common part's
rounding covers the transform's.

Tolerance: the error is the median of the relative errors over the pixels above a
tenth of the median intensity (thousands), whose scatter between two rounding
patterns is a few per cent; 1.25 allows for it.  A mean off by the whole contrast
gives 1.7 (per energy spectra) and 2.6 (fields).  The planes of the film are nearly
constant, and how exactly a constant is transformed follows from its last bits: a
factor of up to 2.3 between neighbouring values of the mean, for which the film's 3
allows; a mean off by the whole contrast gives 6 and more.
"""
import numpy as np
import pytest

from test_gpu_parity import native

pytestmark = pytest.mark.gpu

RATIO, FILM_RATIO = 1.25, 3.0
OPTICAL = np.array([[[4e-3, 0, 4e-3, 0], [-4e-3, 0, -4e-3, 0], [0, 0, 0, 0]]], np.float32)


def _voxels(first):
    vox = np.zeros((3,) + first.shape + (4,), np.float32)
    vox[0, ..., 3] = first
    vox[1, ..., 3] = 1.0 - vox[0, ..., 3]
    return vox


def _error(first, strategy, device):
    nat = native()
    import torch

    nz, ny, nx = first.shape
    opts = nat.Options(nx=nx, ny=ny, nz=nz, num_material=3, energies=[285.0], start_angle=0.0, end_angle=120.0,
                       increment_angle=60.0, phys_size=5.0, rot_mask=1, strategy=strategy)
    vox = _voxels(first)
    want = nat.cuda_main_fp64(opts, OPTICAL, vox)
    if device:
        d_vox, out = torch.from_numpy(vox).cuda(), torch.zeros(want.shape, dtype=torch.float32, device="cuda")
        nat.simulate_device(opts, OPTICAL, d_vox.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
    else:
        got = nat.cuda_main(opts, OPTICAL, vox)
    ok = want > 0.1 * np.median(want[want > 0])  # the peaks of the structure itself are few
    assert ok.sum() > 2000
    return np.median(np.abs(got[ok] - want[ok]) / want[ok])


@pytest.mark.parametrize("strategy", [1, 2])
def test_grating_along_y(strategy):
    rng = np.random.default_rng(16)
    first = 0.3 + 0.002 * rng.standard_normal((16, 512, 512))
    first[:, 0::16] += 0.6
    first[:, 1::16] += 0.6
    errors = [_error(np.roll(first, turn, 1), strategy, True) for turn in (0, 4, 9)]
    assert max(errors) <= RATIO * min(errors), errors


@pytest.mark.parametrize("shape,layers", [((75, 120, 120), (0, 38)), ((64, 128, 128), (0, 32))])
def test_layers_of_a_host_film(shape, layers):
    # 48 MiB of morphology and a bit: two slabs, whose means come from rows copied ahead of them
    rng = np.random.default_rng(17)
    first = 0.5 + 0.002 * rng.standard_normal(shape)
    for z in layers:
        first[z:z + 2] += 0.45
    errors = [_error(np.roll(first, turn, 0), 2, False) for turn in (0, 10, 17, 25)]
    assert max(errors) <= FILM_RATIO * min(errors), errors
