"""Every instance of the FIELDS Ewald kernel against the CPU oracle: LAB frame with 2
and 3 basis vectors and MATERIAL frame, one and two Ewald planes (2D, nearest
neighbour, linear), 1 to 4 materials walked at compile time and 5 with every
term formed, energy counts that end inside a block and a record.

Tolerance: the parity tolerance of tests/test_gpu_parity.py, 1e-4 relative on
pixels above 1e-6 of the peak, and identical NaN masks.
"""
import numpy as np
import pytest

import cases
import oracle
from test_gpu_parity import TOL, native, options_for, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("materials", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("frame", ["lab", "tilted", "material"])
@pytest.mark.parametrize("nz,interp", [(1, cases.LINEAR), (10, cases.NN), (10, cases.LINEAR)])
def test_matches_oracle(materials, frame, nz, interp):
    over = dict(case_type=1, kvecs=[[0.05, 0.02, 1.0]]) if frame == "tilted" else {}
    case = cases.Case("form", 26, 22, nz, materials, [282.0, 284.0, 285.0, 286.0, 289.0], interpolation=interp,
                      seed=40 + materials, geometry="blobs", angles=(0.0, 150.0, 50.0),
                      frame=cases.MATERIAL if frame == "material" else cases.LAB, **over)
    optical, vox = cases.optical_constants(case), cases.voxels(case)
    got = native().cuda_main(options_for(case, strategy=2), optical, vox).astype(np.float64)
    want = oracle.run_case(case)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert rel_err(got, want).max() <= TOL
