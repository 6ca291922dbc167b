"""The surface field against a direct FP64 evaluation over all nodes, where its
kernels change paths: too few neighbours for an ellipsoid, more than one list
of them, particles at the box's edge, tiles cut by the grid's end."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
R_P, R_H = 0.01, 0.02


def _direct(pos, sf, lo, aniso):
    """surface_field.cpp:43-176 in FP64 on the FP32 positions."""
    x = pos.astype(np.float64)
    hf = 2 * R_H
    gmin, num, cell = np.asarray(sf.grid_min, np.float64), np.asarray(sf.grid_num), sf.cell_size
    hn = int(R_H / cell)
    f = np.zeros(tuple(num[::-1]))
    counts = []
    for i in range(len(x)):
        c, G, det, smax = x[i], np.eye(3), 1.0, 1.0
        if aniso:
            d = np.delete(x, i, 0) - x[i]
            r = np.sqrt((d * d).sum(1))
            d, r = d[r <= hf], r[r <= hf]
            counts.append(len(r))
            w = 1 - (r / hf) ** 3
            if len(r) >= 25:
                m = (w[:, None] * d).sum(0) / w.sum()
                C = np.einsum("k,ka,kb->ab", w, d - m, d - m) / w.sum()
                ev, V = np.linalg.eigh(C)
                s = np.abs(ev)
                s = np.maximum(s, s.max() / 4) * (1.6 / (0.16 * hf * hf))
                G, det, smax, c = V @ np.diag(1 / s) @ V.T, 1 / s.prod(), s.max(), x[i] + m
            else:
                k = 0.95 * (3 - 2 * len(r) / 25)
                G, det, smax = np.eye(3) * k, k ** 3, 1 / 0.95
        hw = int(hn * smax) if aniso else hn
        n0 = ((c - gmin) / cell).astype(int)
        a, b = np.maximum(n0 - hw, 0), np.minimum(n0 + hw + 1, num - 1)
        ax = [gmin[k] + cell * np.arange(a[k], b[k] + 1) - c[k] for k in range(3)]
        z, y, u = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        r = np.linalg.norm(np.stack([u, y, z], -1) @ G, axis=-1)
        q = r / R_H
        W = np.where(q < 0.5, 8 - 48 * q ** 2 + 48 * q ** 3, 16 * np.clip(1 - q, 0, None) ** 3) / (math.pi * R_H ** 3)
        f[a[2]:b[2] + 1, a[1]:b[1] + 1, a[0]:b[0] + 1] += det * W * R_P ** 3
    return f, counts


@pytest.mark.parametrize("aniso", [0, 1])
@pytest.mark.parametrize("kind", ["sparse", "block", "dense"])
def test_field_is_the_direct_sum(aniso, kind):
    from graphics_b200.surface import surface_field
    rng = np.random.default_rng(5)
    n, gap = {"sparse": (4, 0.03), "block": (7, 0.02), "dense": (9, 0.0105)}[kind]
    box = 0.145
    lat = (np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * gap
    pos = (lat + rng.uniform(-0.2, 0.2, lat.shape) * gap).astype(np.float32)
    pos[0], pos[1] = 0.0, box  # the box's own corners, few neighbours
    sf = surface_field()
    sf.surface_setup([0.0] * 3, [box] * 3, R_P, R_H, R_P / 2)
    assert (sf.surface_aniso if aniso else sf.surface_isotro)(pos) == 0
    got = sf.get_field().reshape(tuple(np.asarray(sf.grid_num)[::-1]))
    want, counts = _direct(pos, sf, 0.0, aniso)
    if aniso:
        assert {"sparse": max(counts) < 25, "block": 25 < max(counts) <= 56, "dense": max(counts) > 64}[kind]
    # FP32 offsets (2^-24 of 0.15 against distances of 0.02), their products
    # and a sum of up to a hundred kernels of both signs of error
    assert np.max(np.abs(got - want)) <= 2e-5 * np.max(want)
    sf.close()


@pytest.mark.parametrize("ref_rows", [False, True])
@pytest.mark.parametrize("box,share", [((0.15, 0.11, 0.13), 0.5), ((0.07, 0.3, 0.05), 0.02)])
def test_marching_cubes_of_noise_is_the_restatement(ref_rows, box, share):
    """Every cube case, blocks of cubes full of triangles and nearly empty
    ones, rows that end within a thread's cubes: equal bit for bit."""
    import mc_table as mt
    from graphics_b200.surface import surface_field
    sf = surface_field()
    sf.surface_setup([0.0] * 3, box, R_P, R_H, R_P / 2)
    num = [int(v) for v in sf.grid_num]
    rng = np.random.default_rng(3)
    f = rng.uniform(0, 1, num[::-1]).astype(np.float32)
    f[rng.uniform(0, 1, f.shape) > share] += 1
    sf.set_field(f)
    got = sf.mesh(0.9, ref_rows=ref_rows)
    want = mt.marching_cubes(f.ravel(), tuple(num), np.asarray(sf.grid_min, np.float32), np.float32(sf.cell_size), 0.9,
                             ref_rows=ref_rows)
    assert len(want) > 100
    np.testing.assert_array_equal(got, want)
    sf.close()
