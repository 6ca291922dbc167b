"""Solver stages after fields that the caller has set between them (GPU)."""
import numpy as np
import pytest

from graphics_b200.scene import dam_break
from graphics_b200.sph import GpuScene, params_for_scene

pytestmark = pytest.mark.gpu


# WCSPH's plain force pass reads a record per neighbour, which the list build
# writes; the general pass (a second fluid: one particle out of reach in the
# far corner) reads the fields themselves
@pytest.mark.parametrize("lanes", [1, 4])
def test_wcsph_forces_after_set_density(lanes):
    r, counts = 0.0125, (12, 11, 13)
    sc = dam_break(counts, r, tuple(2 * r * (k + 3) for k in counts), seed=4)
    rng = np.random.default_rng(4)
    sc.fluid_vel = rng.normal(0, 0.2, sc.fluid_pos.shape).astype(np.float32)
    factor = rng.uniform(0.8, 1.25, sc.n_fluid + 1).astype(np.float32)
    acc = []
    for far in (0, 1):
        g = GpuScene(params_for_scene(sc, dt=2.5e-4, soundSpeed_cs=18.0, boundary_visc=0.03), sc.n_fluid + 1)
        g.debug_set("wc_lanes", lanes)
        g.set_boundary(sc.boundary_pos)
        g.add_fluid(sc.fluid_pos, sc.fluid_vel, visc_alpha=0.05)
        if far:
            g.add_fluid(np.array([[(k + 2.5) * sc.d for k in counts]], np.float32), rho0=2000.0, visc_alpha=0.05)
        g.stage("wc_computePressure")
        before = g.get("density")
        g.set("density", before * factor[:len(before)])
        np.testing.assert_array_equal(g.get("density"), before * factor[:len(before)])
        g.stage("wc_computeForce")
        acc.append(g.get("acceleration")[:sc.n_fluid])
        g.close()
    # some 50 terms, each a few ulp of the largest, in either pass: 50 * 4 * 2^-24
    assert np.abs(acc[0] - acc[1]).max() <= 50 * 4 * 2.0 ** -24 * np.abs(acc[0]).max()


# the list build of the pressure stage, by a thread and by a warp for a few
# particles: lists, densities and pressures, also over the cap (a block squeezed
# to two thirds) and with a short one
@pytest.mark.parametrize("squeeze,cap", [(1.0, 48), (0.66, 48), (1.0, 10)])
def test_wcsph_pressure_stage_by_either_list_build(squeeze, cap):
    r, counts = 0.0125, (12, 11, 13)
    sc = dam_break(counts, r, tuple(2 * r * (k + 3) for k in counts), seed=5)
    out = []
    for build in (0, 1):
        g = GpuScene(params_for_scene(sc, dt=2.5e-4, soundSpeed_cs=18.0, max_neighbours=cap), sc.n_fluid)
        g.debug_set("build", build)
        g.set_boundary(sc.boundary_pos)
        g.add_fluid((sc.fluid_pos * np.float32(squeeze)).astype(np.float32), sc.fluid_vel)
        g.stage("wc_computePressure")
        count, kind, index = g.neighbours()
        kept = np.arange(kind.shape[1])[None, :] < count[:, None]
        assert count.max() == cap if squeeze < 1 or cap < 48 else count.max() < cap
        out.append((count, kind[kept], index[kept], g.get("density"), g.get("presure")))
        g.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


# One chain of all neighbours leaves an rms error of 1.448e-7 of the density on
# these blocks (measured against FP64).  An addition that brings the sum to the
# fraction f of its end adds about f^2 (2^-24)^2 0.54 / 3 to the square of it: over
# 33 neighbours 11.9 such f^2 in one chain, 3.5 in blocks of eight, a difference
# of 5.4e-15.  The bound is half of that below one chain's.
ONE_CHAIN, GAIN = 1.448e-7, 5.4e-15


@pytest.mark.parametrize("build", [0, 1])
def test_wcsph_density_error_is_that_of_blocked_sums(build):
    from oracle import make_scene_oracle
    err = []
    for seed in range(8):
        r, counts = 0.0125, (11, 10, 12)
        sc = dam_break(counts, r, tuple(2 * r * (k + 3) for k in counts), seed=seed)
        kw = dict(dt=2.5e-4, soundSpeed_cs=18.0)
        g = GpuScene(params_for_scene(sc, **kw), sc.n_fluid)
        g.debug_set("build", build)
        g.set_boundary(sc.boundary_pos)
        g.add_fluid(sc.fluid_pos, sc.fluid_vel)
        g.stage("wc_computePressure")
        o = make_scene_oracle(sc, f64=True, **kw)
        for stage in ("neighbourSearch", "updateSolidPartWeight", "wc_computePressure"):
            o.stage(stage)
        exact = np.asarray(o.get("density"), np.float64)
        err.append(np.sqrt(np.mean((g.get("density") / exact - 1.0) ** 2)))
        g.close()
    assert np.mean(err) < np.sqrt(ONE_CHAIN ** 2 - GAIN / 2)
