"""The mixed-radix and Bluestein passes (k_mix_fft) against numpy, along every
axis: each radix alone, two to five stages, odd and even last radices (with
and without the row form's padding), partial tiles of columns and rows, the
longest lines, lengths with prime factors 11 and 13 and above, and a column
count of one tile and one more.

Tolerance: the FFT parity tolerance of tests/test_gpu_parity.py, 2e-6 of the
largest bin.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-6
SHORT = [2, 3, 4, 5, 6, 7, 9, 10, 11, 12, 13, 14, 15]  # one stage
TWO = [18, 20, 21, 22, 26, 33, 36, 49, 60, 75, 90, 96, 100, 121, 143, 168, 169, 180, 210, 225, 240]
MORE = [250, 264, 343, 360, 441, 450, 500, 1001, 1536, 2048, 2187, 3125, 4096, 6250, 6400]
PRIME = [17, 19, 34, 61, 113, 127, 211, 257, 509, 1021, 2039, 2047]  # a prime factor above 13: Bluestein


def _check(shape, count):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cyrsoxs_gb300 import _native

    rng = np.random.default_rng(sum(shape) + count)
    a = (rng.standard_normal((count,) + shape) + 1j * rng.standard_normal((count,) + shape)).astype(np.complex64)
    d = torch.from_numpy(a.view(np.float32)).cuda()
    nz, ny, nx = shape
    _native.fft3d_device(d.data_ptr(), nx, ny, nz, count, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = d.cpu().numpy().view(np.complex64)
    ref = np.fft.fftn(a.astype(np.complex128), axes=(1, 2, 3))
    err = np.abs(got - ref).max() / np.abs(ref).max()
    assert err < TOL, (shape, err)


@pytest.mark.parametrize("n", SHORT + TWO + MORE + PRIME)
def test_each_axis(n):
    for shape, count in (((3, 5, n), 2), ((3, n, 5), 2), ((n, 3, 5), 2)):
        _check(shape, count)


@pytest.mark.parametrize("n", [15, 18, 90, 240, 61])
@pytest.mark.parametrize("cols", [31, 32, 33, 257])
def test_partial_tiles(n, cols):
    _check((2, n, cols), 1)
    _check((n, 3, cols), 3)
    _check((cols, 3, n), 1)


def test_many_blocks():
    # enough tiles that no block is narrowed, on every axis at once
    _check((60, 210, 240), 3)
    _check((61, 113, 127), 3)
