"""A captured graph serves only requests whose options are the same to the last bit:
k vectors, detector warps and Ewald geometry are part of the captured launches.  Two
signatures that differ by one unit in the last place of a k component or an energy
(equal in the first six decimals) get a graph each, and each request equals itself
run uncaptured.

Tolerance of the comparison: the parity tolerance of tests/test_gpu_parity.py, 1e-4
relative on pixels above 1e-6 of the peak, and identical NaN masks.
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import TOL, native, options_for, rel_err

pytestmark = pytest.mark.gpu


def _options(what):
    """Two options one bit apart, and the case they belong to."""
    k = cases._normalize32([0.05, 0.02, 1.0])
    case = cases.Case("signature", 64, 64, 16, 2, [283.0, 285.0], seed=5, geometry="blobs", angles=(0.0, 150.0, 30.0),
                      case_type=1, kvecs=[k.tolist()])
    near = k.copy()
    energies = np.array(case.energies, np.float32)
    if what == "k":
        near[1] = np.nextafter(near[1], np.float32(1))
    else:
        # energies this small agree to six decimals when one unit in the last place apart
        energies = np.array([0.3, 0.5], np.float32)
    other = energies.copy()
    if what == "energy":
        other[0] = np.nextafter(other[0], np.float32(1))
    return case, [options_for(case, strategy=2, k_vectors=[v.tolist()], energies=e)
                  for v, e in ((k, energies), (near, other))]


@pytest.mark.parametrize("what", ["k", "energy"])
def test_one_graph_per_signature(what):
    nat = native()
    import torch

    from cyrsoxs_gb300 import serving

    case, opts = _options(what)
    optical, vox = cases.optical_constants(case), np.ascontiguousarray(cases.voxels(case), np.float32)
    d_vox = torch.from_numpy(vox).cuda()
    want = [nat.cuda_main(o, optical, vox).astype(np.float64) for o in opts]
    out = torch.zeros(want[0].shape, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    with serving.Server(slots=1, graphs=True) as srv:
        for _ in range(3):  # run, capture, replay
            for o, w in zip(opts, want):
                srv.wait(srv.submit(o, optical, d_vox.data_ptr(), out.data_ptr(), device=True))
                got = out.cpu().numpy().astype(np.float64)
                assert np.array_equal(np.isnan(got), np.isnan(w))
                if not np.isnan(w).all():
                    assert rel_err(got, w).max() <= TOL
        assert srv.stats()["graph_captures"] == 2
