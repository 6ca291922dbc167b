"""Handles after a call that failed, for want of memory or on its input (GPU)."""
import numpy as np
import pytest

from graphics_b200 import _lib
from graphics_b200.scene import small_dam_break
from graphics_b200.sph import GpuScene, SphGpuError, params_for_scene, scene_to_gpu

pytestmark = pytest.mark.gpu


def test_a_failed_handle_does_not_fail_others():
    """A billion particles' arrays are several times the device's memory; the
    scene that is there steps on, as without the attempt."""
    sc = small_dam_break((9, 8, 7), r=0.025, seed=2)
    out = []
    for attempt in (False, True):
        g = scene_to_gpu(sc, dt=1e-3, nu=1e-3)
        g.step("dfsph", 1)
        if attempt:
            with pytest.raises(SphGpuError) as e:
                GpuScene(params_for_scene(sc, dt=1e-3), 1_000_000_000)
            assert e.value.code == _lib.ENOMEM
        g.step("dfsph", 2)
        g.stage("neighbourSearch")
        out.append((g.get("position"), g.get("density")))
        g.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("solver", ["dfsph", "wcsph", "pcisph", "iisph"])
def test_refused_walls_leave_the_ones_that_are_there(solver):
    """Fewer walls than before, one of them outside the grid: an error, and the
    scene goes on with its own."""
    sc = small_dam_break((9, 8, 7), r=0.025, seed=2)
    out = []
    for attempt in (False, True):
        g = scene_to_gpu(sc, dt=5e-4, nu=1e-3, soundSpeed_cs=20.0)
        g.step(solver, 1)
        if attempt:
            few = np.array([[0.01, 0.01, 0.01], [100.0, 0.0, 0.0], [0.02, 0.01, 0.01]], np.float32)
            with pytest.raises(SphGpuError) as e:
                g.set_boundary(few)
            assert e.value.code == _lib.EINVAL
        g.step(solver, 2)
        out.append((g.get("position"), g.get("density"), g.get_boundary("position"), g.get_boundary("volume")))
        g.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
