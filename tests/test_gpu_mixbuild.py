"""The field build fused with the mixed-radix x pass (k_build_fields_mix) against the
CPU oracle: row lengths of two to four stages, with odd and even last radices
(with and without the padded line order), fewer rows than a block takes and a
last tile of rows that is not full, 1 to 5 materials (5: the run-time walk),
both morphology types, with and without a window.

Tolerance: the parity tolerance of tests/test_gpu_parity.py, 1e-4 relative on
pixels above 1e-6 of the peak, and identical NaN masks.
"""
import numpy as np
import pytest

import cases
import oracle
from test_gpu_parity import TOL, native, options_for, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,materials,morphology", [
    (18, 1, cases.EULER), (20, 2, cases.VECTOR), (36, 3, cases.EULER), (64, 4, cases.VECTOR), (90, 5, cases.EULER),
    (143, 2, cases.EULER), (168, 1, cases.VECTOR), (240, 5, cases.VECTOR), (256 + 44, 2, cases.EULER),
    (441, 3, cases.VECTOR), (500, 4, cases.EULER), (768, 2, cases.VECTOR), (1250, 1, cases.EULER)])
@pytest.mark.parametrize("window", [0, 1])
def test_matches_oracle(nx, materials, morphology, window):
    case = cases.Case("mixbuild", nx, 22, 5, materials, [284.0, 286.0], morphology=morphology, windowing=window,
                      seed=nx, geometry="blobs", angles=(0.0, 120.0, 60.0), rot_mask=1)  # unmasked, nothing is left
    optical, vox = cases.optical_constants(case), cases.voxels(case)
    nat = native()
    nat.profile_begin()
    got = nat.cuda_main(options_for(case, strategy=2), optical, vox).astype(np.float64)
    launched, _ = nat.profile_end()
    assert "k_build_fields_rows" in launched
    want = oracle.run_case(case)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert rel_err(got, want).max() <= TOL
