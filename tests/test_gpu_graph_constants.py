"""A captured graph is replayed with other optical constants than it was captured
with.  The order in which the field build walks the materials follows from the
constants (the material whose isotropic contrast lies nearest to the others
comes last), so it must come from the request at every replay.  Two requests
of one signature have their materials' constants exchanged; each is served
several times, so that both run on the other's graph, and must equal
itself alone.

Tolerance: the parity tolerance of tests/test_gpu_parity.py, 1e-4 relative on
pixels above 1e-6 of the peak, and identical NaN masks.
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import TOL, native, options_for, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [False, True])
def test_replay_takes_the_request_s_material_order(groups):
    nat = native()
    import torch

    from cyrsoxs_gb300 import serving

    case = cases.Case("order", 64, 64, 16, 3, [283.0, 285.0], seed=77, geometry="blobs", angles=(0.0, 150.0, 30.0))
    opts, vox = options_for(case, strategy=2), np.ascontiguousarray(cases.voxels(case), np.float32)
    first = cases.optical_constants(case)
    optical = [first, np.ascontiguousarray(first[:, ::-1]), np.ascontiguousarray(np.roll(first, 1, axis=1))]
    want = [nat.cuda_main(opts, o, vox).astype(np.float64) for o in optical]
    d_vox = torch.from_numpy(vox).cuda()
    outs = [torch.zeros(want[0].shape, dtype=torch.float32, device="cuda") for _ in range(9)]
    with serving.Server(slots=1, graphs=True, groups=groups) as srv:
        for k, out in enumerate(outs):
            srv.wait(srv.submit(opts, optical[k % 3], d_vox.data_ptr(), out.data_ptr(), device=True))
        assert srv.stats()["graph_replays"] > 3
        ids = [srv.submit(opts, optical[k % 3], d_vox.data_ptr(), out.data_ptr(), device=True)
               for k, out in enumerate(outs)]  # queued together: a group when groups are on
        for i in ids:
            srv.wait(i)
    for k, out in enumerate(outs):
        got = out.cpu().numpy().astype(np.float64)
        assert np.array_equal(np.isnan(got), np.isnan(want[k % 3]))
        assert rel_err(got, want[k % 3]).max() <= TOL, k
