"""Per-energy spectra of Euler morphologies on both sides of the rule that converts
the morphology once to the trigonometry-free form: by the number of builds, the
material count and the form of the z transform.  The profile shows which side ran (a
converted request launches the build kernel's pair, of which one returns at entry).

Tolerance: the parity tolerance of tests/test_gpu_parity.py, 1e-4 relative on pixels
above 1e-6 of the peak, and identical NaN masks, against the CPU oracle.
"""
import numpy as np
import pytest

import cases
import oracle
from test_gpu_parity import TOL, native, options_for, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,materials,energies,converted", [
    (128, 1, 3, False), (128, 1, 4, True), (128, 3, 4, True), (20, 1, 14, False), (20, 2, 11, False), (20, 3, 12, True),
    (20, 4, 5, False), (20, 4, 6, True), (23, 5, 6, True)])
def test_both_sides_match_oracle(nz, materials, energies, converted):
    case = cases.Case("conversion", 22, 18, nz, materials, [float(e) for e in np.linspace(280.0, 290.0, energies)],
                      seed=nz + materials, geometry="blobs", angles=(0.0, 120.0, 60.0), rot_mask=1)
    optical, vox = cases.optical_constants(case), cases.voxels(case)
    nat = native()
    opts = options_for(case, strategy=1)
    nat.cuda_main(opts, optical, vox)  # tunes the shape
    nat.profile_begin()
    got = nat.cuda_main(opts, optical, vox).astype(np.float64)
    launched, _ = nat.profile_end()
    launches, _, calls = launched["k_build" if nz == 23 else "k_build_fft_z"]
    assert launches == calls * (2 if converted else 1)
    want = oracle.run_case(case)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert rel_err(got, want).max() <= TOL
