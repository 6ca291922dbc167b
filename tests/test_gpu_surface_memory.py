"""The surface handle's growing buffers (GPU): a call that found no memory
leaves a handle that works on."""
import numpy as np
import pytest

from graphics_b200 import _lib
from graphics_b200.sph import SphGpuError

pytestmark = pytest.mark.gpu


class _Full:
    """All of the device's free memory but some 64 MB, while it lasts."""

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        self.held = []
        left = torch.cuda.mem_get_info()[0] - (64 << 20)
        while left >= 1 << 20:
            try:
                self.held.append(torch.empty(left, dtype=torch.uint8, device="cuda"))
                left = torch.cuda.mem_get_info()[0] - (64 << 20)
            except torch.cuda.OutOfMemoryError:
                left //= 2

    def __exit__(self, *a):
        import torch
        self.held.clear()
        torch.cuda.empty_cache()


def _handle(box=0.2):
    from graphics_b200.surface import surface_field
    sf = surface_field()
    sf.surface_setup([0.0] * 3, [box] * 3, 0.01, 0.02, 0.0025)
    return sf


@pytest.mark.parametrize("aniso", [0, 1])
def test_field_after_no_memory_for_particles(aniso):
    import torch
    rng = np.random.default_rng(1)
    many = torch.rand((4_000_000, 3), device="cuda") * 0.2
    pos = rng.uniform(0, 0.2, (3000, 3)).astype(np.float32)
    fresh, sf = _handle(), _handle()
    out = []
    for h in (fresh, sf):
        field = h.surface_aniso if aniso else h.surface_isotro
        assert field(pos) == 0  # the buffers hold 3000
        if h is sf:
            with _Full():
                with pytest.raises(SphGpuError) as e:
                    field(many.data_ptr(), on_device=True, n=len(many))
            assert e.value.code == _lib.ENOMEM
        assert field(pos[:2000]) == 0
        out.append(h.get_field())
    np.testing.assert_array_equal(*out)
    fresh.close()
    sf.close()


def test_mesh_after_no_memory_for_triangles():
    rng = np.random.default_rng(2)
    sf = _handle(0.5)
    num = np.asarray(sf.grid_num)
    f = rng.uniform(0, 1, tuple(num[::-1])).astype(np.float32)
    few = np.where(np.arange(f.shape[0])[:, None, None] < 3, f, np.float32(2.0))
    sf.set_field(few)
    want = sf.mesh(0.5)
    sf.set_field(f)  # some 2.5 triangles of 36 bytes per cube: over 600 MB
    with _Full():
        with pytest.raises(SphGpuError) as e:
            sf.mesh(0.5)
    assert e.value.code == _lib.ENOMEM
    sf.set_field(few)
    np.testing.assert_array_equal(sf.mesh(0.5), want)
    sf.close()


def test_more_than_2_31_triangles():
    """A checkerboard of 814^3 nodes: four lone corners, so four triangles, in
    every cube (77 GB of them on the device)."""
    import ctypes as C
    import torch
    from graphics_b200.surface import surface_field
    if torch.cuda.mem_get_info()[0] < 100e9:
        pytest.skip("needs 100 GB of device memory")
    heads = []
    for n in (34, 814):
        sf = surface_field()
        sf.surface_setup([0.0] * 3, [0.01 * (n - 1) - 0.025] * 3, 0.01, 0.02, 0.01)
        assert [int(v) for v in sf.grid_num] == [n] * 3
        i = (np.arange(n) & 1).astype(np.uint8)
        f = (i[:, None, None] ^ i[None, :, None] ^ i[None, None, :]).astype(np.float32)
        sf.set_field(f)
        head = np.zeros((8, 3, 3), np.float32)
        total = sf.lib.sphgpu_surface_mesh(sf.h, 0.5, 0, head.ctypes.data_as(C.POINTER(C.c_float)), len(head))
        sf.close()
        assert total == 4 * (n - 1) ** 3
        heads.append(head)
    np.testing.assert_array_equal(*heads)


def test_more_than_2_31_tile_pairs_are_refused():
    """300 000 particles at one place, each over more than 8000 tiles; the
    handle then makes another field."""
    from graphics_b200.surface import surface_field
    sf = surface_field()
    sf.surface_setup([0.0] * 3, [0.02] * 3, 0.01, 0.02, 0.02 / 128)
    one = np.full((1, 3), 0.01, np.float32)
    assert sf.surface_isotro(one) == 0
    want, pairs = sf.get_field(), sf.stats()[0]
    n = 300_000
    assert n * pairs > 2 ** 31
    with pytest.raises(SphGpuError) as e:
        sf.surface_isotro(np.repeat(one, n, 0))
    assert e.value.code == _lib.EINVAL
    assert sf.surface_isotro(one) == 0
    np.testing.assert_array_equal(sf.get_field(), want)
    sf.close()
