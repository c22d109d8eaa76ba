"""cyr_required_device_bytes counts the converted copy of an Euler morphology (16 bytes
a voxel and material) only for the requests that make one, on the host alone.  A
vector morphology of the same options never does.
"""
import pytest

from test_boundary import _native


@pytest.mark.parametrize("nz,materials,energies,converted", [
    (128, 2, 1, False), (128, 2, 3, False), (128, 2, 4, True), (90, 1, 100, False), (90, 2, 11, False), (90, 2, 12, True),
    (90, 4, 5, False), (90, 4, 6, True)])
def test_converted_copy(nz, materials, energies, converted):
    nat = _native()

    def needed(morphology, strategy):
        return nat.required_device_bytes(nat.Options(
            nx=64, ny=64, nz=nz, num_material=materials, energies=[280.0 + 0.1 * e for e in range(energies)],
            start_angle=0.0, end_angle=90.0, increment_angle=30.0, phys_size=5.0, morphology_type=morphology,
            strategy=strategy))

    copy = 16 * 64 * 64 * nz * materials
    assert needed(0, 1) - needed(1, 1) == (copy if converted else 0)
    assert needed(0, 2) == needed(1, 2)
