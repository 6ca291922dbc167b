"""Small-scene kernels against the ones larger scenes use (GPU): the results
are the same bit for bit, since both sum in list order."""
import numpy as np
import pytest

from graphics_b200.scene import dam_break, rayleigh_taylor
from graphics_b200.sph import GpuScene, batch_to_gpu, params_for_scene, scene_to_gpu

pytestmark = pytest.mark.gpu

DF = dict(cfl=1, dt_max=1e-3, dt=1e-3, nu=1e-3, df_div_goal_abs=0.0, df_div_goal_rel=1e-3, df_density_max_iter=60)
KW = {"dfsph": DF, "wcsph": dict(dt=2.5e-4, soundSpeed_cs=18.0), "pcisph": dict(dt=1e-3, soundSpeed_cs=20.0),
      "iisph_m": dict(dt=1e-3, soundSpeed_cs=20.0), "iisph": dict(dt=1e-3)}


def _scene(kind, counts, seed=3):
    """A block at rest spacing; "pile": squeezed to two thirds, so that a
    particle sees hundreds of candidates and more neighbours than the cap."""
    r = 0.0125
    if kind == "column":
        return rayleigh_taylor(counts, r, tuple(2 * r * (k + 1) for k in counts), seed=seed)
    sc = dam_break(counts, r, tuple(2 * r * (k + 3) for k in counts), seed=seed)
    if kind == "pile":
        sc.fluid_pos = (sc.fluid_pos * np.float32(0.66)).astype(np.float32)
    sc.fluid_vel = np.random.default_rng(seed).normal(size=sc.fluid_pos.shape).astype(np.float32) * np.float32(0.2)
    return sc


def _run(sc, solver, knob, value, steps=2, **kw):
    g = scene_to_gpu(sc, **{**KW[solver], **kw})
    g.debug_set("wc_lanes", 1)
    g.debug_set(knob, value)
    st = g.step(solver, steps)
    out = {"pos": g.get("position"), "vel": g.get("velocity"), "rho": g.get("density"),
           "count": g.get("neighbour_count"),
           "stats": np.array([st[k] for k in ("iter_density", "iter_divergence", "neighbour_overflow", "status",
                                              "max_neighbours_seen", "mean_neighbours")])}
    if solver == "dfsph":
        out["lists"] = np.concatenate([a.ravel() for a in g.neighbours()])
        out["alpha"], out["kv"] = g.get("DFalpha"), g.get("DFkappaV")
    g.close()
    return out


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


# one particle, fewer than a warp's group, remainders of groups and blocks,
# several particles per warp; over the cap; more than one candidate window
@pytest.mark.parametrize("solver,kind,counts,kw", [
    ("dfsph", "block", (1, 1, 1), {}),
    ("dfsph", "block", (3, 5, 2), {}),
    ("dfsph", "block", (17, 19, 23), {}),
    ("dfsph", "block", (33, 31, 29), {}),
    ("dfsph", "pile", (12, 12, 12), {}),
    ("dfsph", "block", (9, 9, 9), dict(max_neighbours=11)),
    ("wcsph", "block", (13, 11, 12), {}),
    ("wcsph", "pile", (9, 10, 11), {}),
    ("pcisph", "column", (11, 9, 13), {}),
    ("iisph_m", "column", (12, 8, 9), {}),
    ("iisph", "column", (10, 9, 11), {}),
    ("iisph", "block", (14, 13, 15), {}),
])
def test_warp_list_build_is_the_thread_build(solver, kind, counts, kw):
    sc = _scene(kind, counts)
    steps = 1 if kind == "pile" else 2
    _same(_run(sc, solver, "build", 0, steps, **kw), _run(sc, solver, "build", 1, steps, **kw))


def test_warp_list_build_in_a_batch():
    scs = [_scene("block", c, seed=k) for k, c in enumerate([(9, 7, 8), (4, 4, 4), (15, 9, 11)])]
    out = []
    for value in (0, 1):
        b = batch_to_gpu(scs, **DF)
        b.debug_set("build", value)
        b.step("dfsph", 2)
        out.append({"pos": b.get("position"), "vel": b.get("velocity"), "rho": b.get("density")})
        b.close()
    _same(*out)


# rows of one entry to full rows, groups of four and their remainders, walls;
# over the cap; both block sizes
@pytest.mark.parametrize("kind,counts,kw", [
    ("block", (1, 1, 1), {}),
    ("block", (2, 3, 1), {}),
    ("block", (13, 11, 7), {}),
    ("block", (26, 31, 29), {}),
    ("pile", (11, 12, 9), {}),
    ("block", (9, 9, 9), dict(max_neighbours=10)),
])
def test_four_thread_sweeps_are_the_one_thread_sweeps(kind, counts, kw):
    sc = _scene(kind, counts)
    steps = 1 if kind == "pile" else 2
    _same(_run(sc, "dfsph", "sweep_lanes", 1, steps, **kw), _run(sc, "dfsph", "sweep_lanes", 4, steps, **kw))


def test_four_thread_sweeps_in_a_batch():
    scs = [_scene("block", c, seed=k) for k, c in enumerate([(9, 7, 8), (4, 4, 4), (15, 9, 11)])]
    out = []
    for value in (1, 4):
        b = batch_to_gpu(scs, **DF)
        b.debug_set("sweep_lanes", value)
        b.step("dfsph", 2)
        out.append({"pos": b.get("position"), "vel": b.get("velocity"), "rho": b.get("density")})
        b.close()
    _same(*out)


# WCSPH's plain force pass (one record per neighbour) against the general
# one, which a scene of two fluids takes: here the second is one particle out
# of reach in the far corner; both thread counts
@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("counts", [(1, 1, 1), (2, 3, 2), (13, 11, 12)])
def test_wcsph_plain_forces_match_the_general_pass(lanes, counts):
    sc = _scene("block", counts)
    acc = []
    for far in (False, True):
        g = GpuScene(params_for_scene(sc, **KW["wcsph"], boundary_visc=0.03), sc.n_fluid + 1)
        g.debug_set("wc_lanes", lanes)
        g.set_boundary(sc.boundary_pos)
        g.add_fluid(sc.fluid_pos, sc.fluid_vel, visc_alpha=0.05)
        if far:
            corner = np.array([[(k + 2.5) * sc.d for k in counts]], np.float32)
            g.add_fluid(corner, rho0=2000.0, visc_alpha=0.05)
        g.step("wcsph", 1)
        acc.append(g.get("acceleration")[:sc.n_fluid])
        g.close()
    # some 50 terms, each a few ulp of the largest, in either pass: 50 * 4 * 2^-24
    assert np.abs(acc[0] - acc[1]).max() <= 50 * 4 * 2.0 ** -24 * np.abs(acc[0]).max()


# fewer cell keys than a round of the scan, several rounds with a remainder
@pytest.mark.parametrize("counts", [(3, 3, 3), (29, 31, 33)])
def test_one_block_scan_of_the_cell_counts(counts):
    sc = _scene("block", counts)
    _same(_run(sc, "dfsph", "scan", 0), _run(sc, "dfsph", "scan", 1))
