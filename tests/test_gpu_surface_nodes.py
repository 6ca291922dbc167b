"""The surface field where grid nodes fall on the kernels' centres: an
unjittered lattice at multiples of the cell (GPU)."""
import numpy as np
import pytest

from test_gpu_surface_kernels import R_H, R_P, _direct

pytestmark = pytest.mark.gpu


# 0.025: fewer than 25 neighbours within 2 r_h (spheres), 0.015: 80 (ellipsoids
# whose means are the particles, by symmetry); none of the lattice's distances
# is 2 r_h itself
@pytest.mark.parametrize("aniso", [0, 1])
@pytest.mark.parametrize("gap", [0.015, 0.025])
def test_field_on_a_lattice_of_nodes(aniso, gap):
    from graphics_b200.surface import surface_field
    n = 8
    lat = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (0.01 + gap * lat).astype(np.float32)
    sf = surface_field()
    sf.surface_setup([0.0] * 3, [0.02 + gap * (n - 1)] * 3, R_P, R_H, R_P / 2)
    assert (sf.surface_aniso if aniso else sf.surface_isotro)(pos) == 0
    got = sf.get_field().reshape(tuple(np.asarray(sf.grid_num)[::-1]))
    assert np.isfinite(got).all()
    want, _ = _direct(pos, sf, 0.0, aniso)
    # FP32 offsets (2^-24 of 0.15 against distances of 0.02), their products
    # and a sum of up to a hundred kernels of both signs of error
    assert np.max(np.abs(got - want)) <= 2e-5 * np.max(want)
    sf.close()
