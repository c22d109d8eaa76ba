"""The rotation's three forms: k_rotate_gram on 32 x 32 and on 16 x 16 tiles, and
k_rotate_direct.  The number of record groups in a launch picks the form, so a
request of many energies (tiles) is compared, energy by energy, with requests
of one energy (direct), on image sizes that end inside a tile, square and not,
with 2 and 3 basis vectors, with and without the rotation mask; and with the
CPU oracle.

Tolerance: the parity tolerance of tests/test_gpu_parity.py, 1e-4 relative on
pixels above 1e-6 of the peak, and identical NaN masks.
"""
import dataclasses

import numpy as np
import pytest

import cases
import oracle
from test_gpu_parity import native, options_for, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-4
TILTED = dict(case_type=1, kvecs=[[0.05, 0.02, 1.0]])


def _case(nx, ny, ne, mask, tilted):
    return cases.Case("rotation", nx, ny, 4, 2, [float(e) for e in np.linspace(280.0, 290.0, ne)], seed=7,
                      geometry="blobs", angles=(0.0, 150.0, 37.5), rot_mask=mask, **(TILTED if tilted else {}))


def _run(case, optical, vox):
    opts = options_for(case, strategy=2)
    return native().cuda_main(opts, optical, vox).astype(np.float64)


@pytest.mark.parametrize("mask", [0, 1])
@pytest.mark.parametrize("tilted", [False, True])
@pytest.mark.parametrize("nx,ny,ne", [(250, 243, 64), (100, 84, 64), (49, 33, 7)])
def test_tiles_equal_direct_and_oracle(nx, ny, ne, mask, tilted):
    case = _case(nx, ny, ne, mask, tilted)
    optical, vox = cases.optical_constants(case), cases.voxels(case)
    got = _run(case, optical, vox)
    for e in (0, ne // 2, ne - 1):
        one = dataclasses.replace(case, energies=[case.energies[e]])
        want = _run(one, optical[e:e + 1], vox)[0]
        assert np.array_equal(np.isnan(got[e]), np.isnan(want))
        assert rel_err(got[e], want).max() <= TOL
    want, _ = oracle.run_arrays(nx=nx, ny=ny, nz=case.nz, energies=[case.energies[ne // 2]],
                                optical=optical[ne // 2:ne // 2 + 1], voxels=vox, angles=case.angles,
                                phys_size=case.phys_size, rot_mask=mask, case_type=case.case_type, kvecs=case.kvecs)
    assert np.array_equal(np.isnan(got[ne // 2]), np.isnan(want[0]))
    assert rel_err(got[ne // 2], want[0]).max() <= TOL
