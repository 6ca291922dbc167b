"""Handles with room for more particles than they hold, kernels forced where
the rules by size would not take them, and batches of very many scenes (GPU):
per-block sums stay within their buffer, results are the same bit for bit."""
import numpy as np
import pytest

from graphics_b200.scene import dam_break, rayleigh_taylor
from graphics_b200.sph import GpuBatch, GpuScene, SphGpuError, params_for_scene

pytestmark = pytest.mark.gpu

DF = dict(cfl=1, dt_max=1e-3, dt=1e-3, nu=1e-3, df_div_goal_abs=0.0, df_div_goal_rel=1e-3, df_density_max_iter=60)
MULTI = dict(dt=1e-3, soundSpeed_cs=20.0)
KW = {"dfsph": DF, "pcisph": MULTI, "iisph_m": MULTI, "iisph": dict(dt=1e-3)}


def _scene(solver, counts=(11, 9, 10)):
    r = 0.0125
    if solver in ("pcisph", "iisph_m"):
        return rayleigh_taylor(counts, r, tuple(2 * r * (k + 1) for k in counts), seed=2)
    sc = dam_break(counts, r, tuple(2 * r * (k + 3) for k in counts), seed=2)
    sc.fluid_vel = np.random.default_rng(2).normal(size=sc.fluid_pos.shape).astype(np.float32) * np.float32(0.2)
    return sc


def _run(solver, cap=0, knobs=(), steps=2):
    sc = _scene(solver)
    g = GpuScene(params_for_scene(sc, **KW[solver]), max(cap, sc.n_fluid))
    g.set_boundary(sc.boundary_pos)
    phase = np.zeros(sc.n_fluid, np.int32) if sc.phase is None else sc.phase
    for ph, rho in enumerate(sc.rho0_phases):
        g.add_fluid(sc.fluid_pos[phase == ph], sc.fluid_vel[phase == ph], rho0=rho)
    for k, v in knobs:
        g.debug_set(k, v)
    st = g.step(solver, steps)
    out = {f: g.get(f) for f in ("position", "velocity", "density", "neighbour_count")}
    out["stats"] = np.array([st[k] for k in ("iter_density", "iter_divergence", "dt", "status", "mean_neighbours",
                                             "n_fluid")])
    g.close()
    return out


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


# every kernel that leaves a sum per block, at a capacity whose blocks of 16 or
# 32 particles are more than the capacity's 64ths and 4096
@pytest.mark.parametrize("knobs", [[("sweep_lanes", 4)], [("build", 1)], [("build", 1), ("sweep_lanes", 4)]])
def test_forced_kernels_in_a_large_handle(knobs):
    _same(_run("dfsph"), _run("dfsph", 300_000, knobs))


# capacities on both sides of the sizes at which the kernels change, around one
# and the same thousand particles
@pytest.mark.parametrize("solver,cap", [("dfsph", 12_001), ("dfsph", 24_001), ("dfsph", 65_537), ("pcisph", 65_537),
                                        ("pcisph", 262_145), ("iisph_m", 65_537), ("iisph_m", 262_145),
                                        ("iisph", 65_537)])
def test_capacity_does_not_change_results(solver, cap):
    _same(_run(solver), _run(solver, cap))


# lists by warps and the sums by threads: what handles of 65 537 to 262 144 particles run
@pytest.mark.parametrize("solver", sorted(KW))
def test_lists_alone_by_warps(solver):
    _same(_run(solver, knobs=[("build", 0)]), _run(solver, knobs=[("build", 2)]))


# threads per particle of WCSPH's force pass (they differ in the order of the
# sums): the plain pass, two fluids, surface terms, on both sides of their lines
@pytest.mark.parametrize("kind,cap,lanes", [("plain", 65_536, 4), ("plain", 65_537, 1), ("two", 65_537, 4),
                                            ("two", 262_144, 4), ("two", 262_145, 1), ("surface", 65_537, 4),
                                            ("surface", 262_145, 1)])
def test_threads_per_particle_of_the_wcsph_forces(kind, cap, lanes):
    sc = _scene("pcisph" if kind == "two" else "dfsph")
    kw = dict(dt=2.5e-4, soundSpeed_cs=18.0)
    if kind == "surface":
        kw.update(th_h=sc.smooth_radius, th_r=0.2, th_bt=1.0)
    out = []
    for forced in (0, lanes, 5 - lanes):
        g = GpuScene(params_for_scene(sc, **kw), cap)
        g.debug_set("wc_lanes", forced)
        g.set_boundary(sc.boundary_pos)
        phase = np.zeros(sc.n_fluid, np.int32) if sc.phase is None else sc.phase
        for ph, rho in enumerate(sc.rho0_phases):
            g.add_fluid(sc.fluid_pos[phase == ph], sc.fluid_vel[phase == ph], rho0=rho, visc_alpha=0.05)
        g.step("wcsph", 1)
        out.append(g.get("acceleration"))
        g.close()
    np.testing.assert_array_equal(out[0], out[1])
    assert not np.array_equal(out[0], out[2])


def test_unknown_list_builds_are_refused():
    sc = _scene("dfsph", (2, 2, 2))
    g = GpuScene(params_for_scene(sc, **DF), sc.n_fluid)
    for v in (-2, 3):
        with pytest.raises(SphGpuError):
            g.debug_set("build", v)
    g.close()


def test_a_batch_of_more_scenes_than_blocks():
    """One chunk of sums per scene, 5000 scenes of one or two particles: each
    scene ends where it does among 50."""
    sc = _scene("dfsph", (1, 1, 1))
    rng = np.random.default_rng(7)
    n, box = 5000, 0.1
    two = np.arange(n) % 3 == 0
    scene = np.sort(np.concatenate([np.arange(n), np.arange(n)[two]])).astype(np.int32)
    pos = rng.uniform(0.04, 0.06, (len(scene), 3)).astype(np.float32)
    vel = rng.normal(0, 0.2, pos.shape).astype(np.float32)
    wall = np.full((n, 3), 0.03, np.float32)
    out = []
    for m in (50, n):
        b = GpuBatch(params_for_scene(sc, **DF), np.zeros((m, 3)), np.full((m, 3), box), int((scene < m).sum()))
        b.set_boundary(wall[:m], np.arange(m))
        k = scene < m
        b.add_fluid(pos[k], vel[k], scene[k])
        b.step("dfsph", 2)
        st = b.scene_stats()[:50]
        first = int((scene < 50).sum())
        out.append({"position": b.get("position")[:first], "velocity": b.get("velocity")[:first],
                    "stats": np.array([[s[f] for f in ("n_fluid", "iter_density", "iter_divergence", "err_density",
                                                       "err_divergence", "dt", "status")] for s in st])})
        b.close()
    assert np.isfinite(out[1]["position"]).all()
    _same(*out)
