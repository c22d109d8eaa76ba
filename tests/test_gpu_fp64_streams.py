"""FP64 requests on different streams share the device's FP64 scratch: each must wait
for the one before it, whichever streams they run on and whichever entry point they
come from.  Requests are enqueued back to back without a synchronisation and must
equal, bit by bit, the same requests run one at a time.
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import native, options_for

pytestmark = pytest.mark.gpu


def _requests(torch):
    out = []
    # the first is much the largest, so that the others would overtake it; both strategies
    for i, (nx, ny, nz, ne, strategy) in enumerate([(128, 128, 32, 6, 2), (64, 48, 16, 2, 1), (96, 96, 24, 3, 2),
                                                     (64, 64, 16, 1, 1)]):
        case = cases.Case("streams", nx, ny, nz, 2, [280.0 + 2 * e for e in range(ne)], seed=20 + i, geometry="blobs",
                          angles=(0.0, 150.0, 30.0))
        vox = np.ascontiguousarray(cases.voxels(case), np.float32)
        out.append((options_for(case, strategy=strategy), cases.optical_constants(case), vox, torch.from_numpy(vox).cuda(),
                    case))
    return out


def test_back_to_back_requests_on_several_streams():
    nat = native()
    import torch

    reqs = _requests(torch)

    want = []
    for opts, optical, _, d_vox, case in reqs:  # one at a time
        out = torch.zeros((len(case.energies), 1, case.ny, case.nx), dtype=torch.float64, device="cuda")
        nat.simulate_device_fp64(opts, optical, d_vox.data_ptr(), False, out.data_ptr(),
                                 torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        want.append(out.cpu().numpy())
    streams = [torch.cuda.Stream() for _ in reqs]
    for _ in range(4):
        outs = [torch.zeros(w.shape, dtype=torch.float64, device="cuda") for w in want]
        torch.cuda.synchronize()
        for (opts, optical, _, d_vox, _), out, s in zip(reqs, outs, streams):
            nat.simulate_device_fp64(opts, optical, d_vox.data_ptr(), False, out.data_ptr(), s.cuda_stream)
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert np.array_equal(o.cpu().numpy(), w, equal_nan=True)


def test_host_calls_behind_a_device_call():
    nat = native()
    import torch

    reqs = _requests(torch)
    opts, optical, vox, d_vox, case = reqs[0]
    small, small_optical, small_vox, _, _ = reqs[1]
    want = nat.cuda_main_fp64(opts, optical, vox)
    want_small = nat.cuda_main_fp64(small, small_optical, small_vox)
    want_pol = nat.compute_polarization_fp64(small, small_optical, small_vox, 0.3, 0)
    stream = torch.cuda.Stream()
    for _ in range(4):
        out = torch.zeros(want.shape, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        nat.simulate_device_fp64(opts, optical, d_vox.data_ptr(), False, out.data_ptr(), stream.cuda_stream)
        got_pol = nat.compute_polarization_fp64(small, small_optical, small_vox, 0.3, 0)
        nat.simulate_device_fp64(opts, optical, d_vox.data_ptr(), False, out.data_ptr(), stream.cuda_stream)
        got_small = nat.cuda_main_fp64(small, small_optical, small_vox)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
        assert np.array_equal(got_small, want_small, equal_nan=True)
        assert all(np.array_equal(a, b) for a, b in zip(got_pol, want_pol))
