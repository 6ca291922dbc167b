"""Workloads of the SPH framework, for timing and for comparing results.

A case names a kind of work, a size and the options it runs with; one pass
is what a program that uses the framework does between two looks at its
particles: it hands over positions and velocities, advances a few steps and
takes the particles back (a simulation frame), or it reconstructs a surface,
or trains the warm-start network for an epoch.  Scenes are dam breaks and
two-phase columns of jittered lattices in walled boxes, as in
graphics_b200.scene, moving with a smooth seeded velocity field.
"""
import math

import numpy as np
import torch

from graphics_b200 import scene as scenes
from graphics_b200 import sph
from graphics_b200.surface import surface_field
from graphics_b200.warmstart import NIN, NPARAM, WarmStartNet, attach

DFSPH_KW = dict(cfl=1, cfl_factor=0.4, dt_max=2e-3, dt_min=1e-6, dt=2e-3, nu=1e-3,
                df_density_goal=1e-4, df_density_min_iter=2, df_density_max_iter=1000,
                df_div_goal_abs=0.0, df_div_goal_rel=1e-3, df_div_min_iter=1, df_div_max_iter=100)
WCSPH_KW = dict(dt=2.5e-4, soundSpeed_cs=18.708287, wc_gamma=7.0, cfl=0, boundary_visc=0.01)
MULTI_KW = dict(dt=1e-3, nu=1e-3, soundSpeed_cs=20.0, cfl=0, boundary_visc=0.01)
PCISPH_KW = dict(densityErro_eta=1e-2, pci_min_iter=3, pci_max_iter=10)
IISPH_M_KW = dict(ii_omega=0.5, ii_eta_rel=5e-4, ii_min_iter=2, ii_max_iter=100, ii_compat=0)
VISC = 0.01


def listed():
    return [
        # the weakly compressible dam break: many cheap fixed steps per frame
        dict(name="wcsph_27k", kind="wcsph", nx=30, ny=30, nz=30, r=0.025, steps=20),
        # the smallest interactive scene: bound by launches and latency
        dict(name="dfsph_1k", kind="dfsph", nx=10, ny=10, nz=10, r=0.025, steps=4),
        # an ordinary scene, odd counts on every axis
        dict(name="dfsph_68k", kind="dfsph", nx=45, ny=37, nz=41, r=0.0125, steps=5),
        # the headline dam break
        dict(name="dfsph_1m", kind="dfsph", nx=100, ny=100, nz=100, r=0.01, steps=8),
        # a host program that keeps the arrays (pinned) and hands them back every step
        dict(name="host_loop_343k", kind="dfsph_host", nx=70, ny=70, nz=70, r=0.01, steps=4),
        # the learned warm start: features and network every step
        dict(name="warm_512k", kind="dfsph_warm", nx=80, ny=80, nz=80, r=0.01, steps=4),
        # two-phase columns under the two pressure solvers for them
        dict(name="pcisph_119k", kind="pcisph", nx=63, ny=30, nz=63, r=0.0079365, steps=2),
        dict(name="iisph_m_95k", kind="iisph_m", nx=63, ny=24, nz=63, r=0.0079365, steps=1),
        # the volume form, one fluid
        dict(name="iisph_64k", kind="iisph", nx=40, ny=40, nz=40, r=0.0125, steps=2),
        # independent scenes of uneven size in one handle
        dict(name="batch_12", kind="batch", scenes=12, nmin=10000, nmax=100000, pick=5, steps=3),
        # a mesh of the particles for rendering: anisotropic kernels, marching cubes
        dict(name="surface_46k", kind="surface", nx=36, ny=36, nz=36, r=0.01, aniso=1, div=2),
        # one epoch of the warm-start network
        dict(name="train_512k", kind="train", rows=524288, batch=8192),
    ]


def draw(rng):
    def counts(lo, hi, flat=1.0):
        """Lattice counts of about exp(U(log lo, log hi)) particles, uneven axes."""
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        a = [rng.uniform(0.8, 1.25), rng.uniform(0.8, 1.25) * flat, rng.uniform(0.8, 1.25)]
        s = (n / (a[0] * a[1] * a[2])) ** (1.0 / 3.0)
        return dict(zip(("nx", "ny", "nz"), (max(6, int(round(s * x))) for x in a)))

    radii = (0.008, 0.01, 0.0125, 0.02, 0.025)
    kind = rng.choice(("wcsph", "dfsph", "dfsph", "dfsph", "dfsph_host", "dfsph_warm", "pcisph", "iisph_m", "iisph",
                       "batch", "surface", "train"))
    if kind == "wcsph":
        return dict(kind=kind, **counts(5e3, 6e5), r=0.025, steps=rng.randint(5, 20))
    if kind == "dfsph":
        return dict(kind=kind, **counts(1e3, 9e5), r=rng.choice(radii), steps=rng.randint(2, 6))
    if kind == "dfsph_host":
        return dict(kind=kind, **counts(1e4, 6e5), r=rng.choice(radii), steps=rng.randint(2, 5))
    if kind == "dfsph_warm":
        return dict(kind=kind, **counts(3e4, 7e5), r=rng.choice(radii), steps=rng.randint(2, 5))
    if kind == "pcisph":
        return dict(kind=kind, **counts(1e4, 2e5, 0.45), r=0.0079365, steps=rng.randint(1, 2))
    if kind == "iisph_m":
        return dict(kind=kind, **counts(1e4, 1.5e5, 0.4), r=0.0079365, steps=1)
    if kind == "iisph":
        return dict(kind=kind, **counts(5e3, 2e5), r=rng.choice(radii), steps=rng.randint(1, 2))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(4, 16), nmin=5000, nmax=rng.randint(20000, 90000),
                    pick=rng.randint(0, 999), steps=rng.randint(2, 3))
    if kind == "surface":
        return dict(kind=kind, **counts(8e3, 6e4), r=0.01, aniso=rng.randint(0, 1),
                    div=rng.choice((2, 4)))
    return dict(kind=kind, rows=int(math.exp(rng.uniform(math.log(3e4), math.log(6e5)))),
                batch=rng.choice((2048, 4096, 8192)))


LOOSE = np.float32(1.005)  # lattice blocks a little wider than at rest density: the loops then need what a
#                            moving fluid needs (2 to 20 iterations a step), not what a start from a lattice does


def _velocity(pos, seed):
    """A smooth divergence-free field of about 0.5 m/s: three seeded shear waves."""
    g = np.random.default_rng(seed + 77)
    x = pos.astype(np.float64)
    ext = float(np.ptp(x, axis=0).max())
    v = np.zeros_like(x)
    for _ in range(3):
        k = g.normal(size=3) * (2.0 / ext)
        a = np.cross(k, g.normal(size=3))
        v += a / np.linalg.norm(a) * np.sin(x @ k + g.uniform(0, 2 * math.pi))[:, None]
    return v.astype(np.float32)


def _scene(case, seed):
    kind, r = case["kind"], case["r"]
    counts = (case["nx"], case["ny"], case["nz"])
    d = 2.0 * r
    if kind in ("pcisph", "iisph_m"):
        sc = scenes.rayleigh_taylor(counts, r, tuple((c + 1) * d for c in counts), seed=seed)
    else:
        # walls at twice the block's length along x, a fifth more height and depth
        box = (2 * counts[0] * d, (counts[1] + max(2, counts[1] // 5)) * d, (counts[2] + max(2, counts[2] // 5)) * d)
        sc = scenes.dam_break(counts, r, box, seed=seed)
    sc.fluid_pos = sc.fluid_pos * LOOSE
    sc.fluid_vel = _velocity(sc.fluid_pos, seed)
    return sc


def _batch_scenes(case, seed):
    out = []
    for k, counts in enumerate(_batch_counts(case)):
        d = 0.02  # r = 0.01; a spacing of room beside the block
        sc = scenes.dam_break(counts, 0.01, (2 * counts[0] * d, (counts[1] + 2) * d, (counts[2] + 2) * d),
                              seed=(seed * 1000 + k) % 2 ** 31)
        sc.fluid_pos = sc.fluid_pos * LOOSE
        sc.fluid_vel = _velocity(sc.fluid_pos, seed * 1000 + k)
        out.append(sc)
    return out


def _to_gpu(sc, visc=None, **kw):
    """As sph.scene_to_gpu, with an artificial viscosity per fluid."""
    if visc is None:
        return sph.scene_to_gpu(sc, **kw)
    g = sph.GpuScene(sph.params_for_scene(sc, **kw), sc.n_fluid)
    g.set_boundary(sc.boundary_pos)
    if sc.phase is None:
        g.add_fluid(sc.fluid_pos, sc.fluid_vel, rho0=sc.rho0, visc_alpha=visc)
    else:
        for ph, rho in enumerate(sc.rho0_phases):
            m = sc.phase == ph
            g.add_fluid(sc.fluid_pos[m], sc.fluid_vel[m], rho0=rho, visc_alpha=visc)
    return g


def _phase_order(sc):
    """Positions and velocities in the framework's particle order (phase by phase)."""
    if sc.phase is None:
        return sc.fluid_pos, sc.fluid_vel
    o = np.argsort(sc.phase, kind="stable")
    return np.ascontiguousarray(sc.fluid_pos[o]), np.ascontiguousarray(sc.fluid_vel[o])


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float32, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _network(seed):
    """An untrained network whose predictions stay small."""
    g = np.random.default_rng(seed)
    w = g.normal(size=NPARAM).astype(np.float32) * 0.2
    norm = np.concatenate([np.zeros(NIN), np.ones(NIN), [0.0, 1e9]]).astype(np.float32)
    return w, norm


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "train":
        g = np.random.default_rng(seed)
        X = g.normal(size=(case["rows"], NIN)).astype(np.float32)
        y = (np.tanh(X[:, 0] * 1.5) + 0.3 * X[:, 1] * X[:, 2] + 0.1 * X[:, 3]).astype(np.float32)
        net = WarmStartNet(dataset_cap=case["rows"], seed=seed)
        net.set_norm(np.concatenate([np.zeros(NIN), np.ones(NIN), [0.0, 1.0]]).astype(np.float32))
        net.set_dataset(X, y)
        s.update(net=net, w0=net.params())
        return s
    if kind == "surface":
        r = case["r"]
        pos = scenes.lattice_block((case["nx"], case["ny"], case["nz"]), r, seed=seed)
        sf = surface_field()
        cell = r / case["div"]
        box = [2 * r * case[a] for a in ("nx", "ny", "nz")]  # holds the jittered lattice
        sf.surface_setup([0.0] * 3, box, r, 2 * r, cell)
        # a vertex buffer for the mesh, as a renderer keeps: two triangles per
        # surface cell and room for the ripples
        a, b, c = (x + 4 * r for x in box)
        s.update(sf=sf, pos=torch.from_numpy(pos).cuda(),
                 mesh=np.zeros((int(10 * (a * b + b * c + c * a) / cell ** 2), 3, 3), np.float32))
        return s
    if kind == "batch":
        scs = _batch_scenes(case, seed)
        s.update(g=sph.batch_to_gpu(scs, **DFSPH_KW), solver="dfsph",
                 pos=np.concatenate([sc.fluid_pos for sc in scs]), vel=np.concatenate([sc.fluid_vel for sc in scs]))
        return s
    sc = _scene(case, seed)
    if kind == "wcsph":
        g, solver = _to_gpu(sc, VISC, **WCSPH_KW), "wcsph"
    elif kind == "pcisph":
        g, solver = _to_gpu(sc, VISC, **MULTI_KW, **PCISPH_KW), "pcisph"
    elif kind == "iisph_m":
        g, solver = _to_gpu(sc, VISC, **MULTI_KW, **IISPH_M_KW), "iisph_m"
    elif kind == "iisph":
        g, solver = _to_gpu(sc, **MULTI_KW), "iisph"
    else:
        g, solver = _to_gpu(sc, **DFSPH_KW), "dfsph"
    pos, vel = _phase_order(sc)
    s.update(g=g, solver=solver, pos=pos, vel=vel)
    if kind == "dfsph_host":
        s.update(pos=_pinned(pos), vel=_pinned(vel), pos_out=_pinned(pos), vel_out=_pinned(vel))
    if kind == "dfsph_warm":
        w, norm = _network(seed)
        net = WarmStartNet(dataset_cap=16, seed=seed)
        net.set_params(w)
        net.set_norm(norm)
        attach(g, net, 1)
        s.update(net=net)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        s["net"].set_params(s["w0"])
        loss = s["net"].train(epochs=1, batch=case["batch"])
        return {"params": s["net"].params(), "loss": loss}
    if kind == "surface":
        sf = s["sf"]
        field = sf.surface_aniso if case["aniso"] else sf.surface_isotro
        field(s["pos"].data_ptr(), on_device=True, n=s["pos"].shape[0])
        tris = sf.mesh(0.5)
        s["mesh"][:len(tris)] = tris
        return {"mesh": s["mesh"], "triangles": len(tris)}
    g = s["g"]
    if kind == "dfsph_host":
        # the first step takes the program's state, the next ones what the step before returned
        g.step_host("dfsph", s["pos"], s["vel"], s["pos_out"], s["vel_out"])
        for _ in range(case["steps"] - 1):
            g.step_host("dfsph", s["pos_out"], s["vel_out"], s["pos_out"], s["vel_out"])
        return {"position": s["pos_out"], "velocity": s["vel_out"]}
    g.set("position", s["pos"])
    g.set("velocity", s["vel"])
    st = g.step(s["solver"], case["steps"])
    return {"position": g.get("position"), "velocity": g.get("velocity"), "n_fluid": st["n_fluid"]}


def work(case):
    """Per step and particle: the state read and written once (48 bytes), and
    for each of about 32 neighbours the distance test and the terms of the
    sums that the solver cannot do without (its fewest iterations)."""
    kind = case["kind"]
    if kind == "train":
        # the rows read once; forward and backward of 16-64-64-1
        return {"bytes": 68.0 * case["rows"], "flops": 6.0 * (16 * 64 + 64 * 64 + 64) * case["rows"]}
    if kind == "surface":
        nodes = 1.0
        for a in ("nx", "ny", "nz"):
            nodes *= (2 * case[a] * case["r"] + 3 * case["r"]) * case["div"] / case["r"]
        n = case["nx"] * case["ny"] * case["nz"]
        # nodes within 2 r_p of a particle: (4/3) pi (2 div)^3, 12 operations each
        return {"bytes": 8.0 * nodes + 12.0 * n, "flops": 400.0 * case["div"] ** 3 * n}
    if kind == "batch":
        n = float(sum(a * b * c for a, b, c in _batch_counts(case)))
    else:
        n = float(case["nx"] * case["ny"] * case["nz"])
    per_pair = {"wcsph": 60, "dfsph": 150, "dfsph_host": 150, "dfsph_warm": 180, "pcisph": 200, "iisph_m": 250,
                "iisph": 300, "batch": 150}[kind]
    extra = 10400.0 * n if kind == "dfsph_warm" else 0.0
    return {"bytes": 48.0 * n * case["steps"], "flops": (32.0 * per_pair * n + extra) * case["steps"]}


def _batch_counts(case):
    """Lattice counts of a batch's scenes: sizes log-uniform, aspect ratios
    uniform in [0.5, 2] per axis, as scenes.config_batched_dfsph draws them."""
    rng = np.random.default_rng(case["pick"])
    out = []
    for _ in range(case["scenes"]):
        n = float(np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]))))
        a = rng.uniform(0.5, 2.0, 3)
        a = a / np.prod(a) ** (1.0 / 3.0)
        out.append(tuple(max(2, int(round(n ** (1.0 / 3.0) * a[k]))) for k in range(3)))
    return out


# ---- the same steps in 64 bits, from the method's equations ----

class _Exact:
    """One walled scene of a single fluid in FP64 torch: cubic spline of
    support 2h = 2d, particle mass rho0 d^3, wall volumes from the walls'
    own density."""

    def __init__(self, sc, rho0=1000.0):
        f = lambda a: torch.as_tensor(a, dtype=torch.float32).cuda().double()  # noqa: E731
        self.x, self.v, self.b = f(sc.fluid_pos), f(sc.fluid_vel), f(sc.boundary_pos)
        self.d = float(np.float32(sc.d))
        self.h = float(np.float32(sc.smooth_radius)) / 2
        self.rho0 = rho0
        self.m = rho0 * float(np.float32(sc.spacing_r)) ** 3
        self.g = torch.tensor([0.0, float(np.float32(-9.81)), 0.0], dtype=torch.float64, device="cuda")
        self.vol = None
        i, _, r = self._pairs(self.b, self.b)[:3]
        s = torch.full((len(self.b),), self.W(torch.zeros(1, dtype=torch.float64)).item(), device="cuda",
                       dtype=torch.float64)
        s.index_add_(0, i, self.W(r))
        self.vol = 1.0 / s

    def W(self, r):
        q = r / self.h
        t = 1.0 / (math.pi * self.h ** 3)
        return torch.where(q <= 1, t * (1 - 1.5 * q * q + 0.75 * q ** 3), t * 0.25 * (2 - q).clamp(min=0) ** 3)

    def F(self, r):
        """W'(r) / r"""
        q = r / self.h
        t = 1.0 / (math.pi * self.h ** 4)
        return -torch.where(q <= 1, t * (3 * q - 2.25 * q * q), t * 0.75 * (2 - q).clamp(min=0) ** 2) / r

    def _pairs(self, a, b, same=True):
        """(i, j, r) of all pairs closer than 2d, i in a, j in b."""
        cut = 2 * self.d
        lo = torch.minimum(a.min(0)[0], b.min(0)[0]) - 2 * cut
        num = ((torch.maximum(a.max(0)[0], b.max(0)[0]) - lo) / cut).long() + 3
        cell = lambda x: ((x - lo) / cut).long()  # noqa: E731
        lin = lambda c: (c[:, 2] * num[1] + c[:, 1]) * num[0] + c[:, 0]  # noqa: E731
        kb, order = torch.sort(lin(cell(b)))
        start = torch.searchsorted(kb, torch.arange(int(num.prod()) + 1, device="cuda"))
        ca = cell(a)
        at = torch.arange(len(a), device="cuda")
        I, J, R = [], [], []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                row = lin(ca + torch.tensor([-1, dy, dz], device="cuda"))
                s0, s1 = start[row], start[row + 3]
                for k in range(int((s1 - s0).max())):
                    ok = s0 + k < s1
                    i = at[ok]
                    j = order[s0[ok] + k]
                    r = (a[i] - b[j]).norm(dim=1)
                    keep = (r < cut) & ((i != j) if same else torch.ones_like(ok[:1]))
                    I.append(i[keep]); J.append(j[keep]); R.append(r[keep])
        return torch.cat(I), torch.cat(J), torch.cat(R)

    def search(self):
        n = len(self.x)
        i, j, r = self._pairs(self.x, self.x)
        ib, jb, rb = self._pairs(self.x, self.b, same=False)
        i = torch.cat([i, ib]); r = torch.cat([r, rb])
        wall = torch.zeros(len(i), dtype=torch.bool, device="cuda")
        wall[len(j):] = True
        j = torch.cat([j, jb])
        i, o = torch.sort(i, stable=True)
        j, r, wall = j[o], r[o], wall[o]
        cnt = torch.bincount(i, minlength=n)
        k = torch.arange(len(i), device="cuda") - (cnt.cumsum(0) - cnt)[i]
        shape = (n, int(cnt.max()))
        flat = i * shape[1] + k

        def ell(v, fill):
            out = torch.full((shape[0] * shape[1],), fill, dtype=v.dtype, device="cuda")
            out[flat] = v
            return out.reshape(shape)

        self.ok, self.wall = ell(torch.ones_like(wall), False), ell(wall, False)
        self.r = ell(r, self.h)
        self.j = ell(torch.where(wall, torch.zeros_like(j), j), 0)
        self.bj = ell(torch.where(wall, j, torch.zeros_like(j)), 0)
        xj = torch.where(self.wall[..., None], self.b[self.bj], self.x[self.j])
        self.xij = self.x[:, None] - xj
        self.mj = torch.where(self.wall, self.rho0 * self.vol[self.bj], torch.full_like(self.r, self.m)) * self.ok
        self.fm = self.F(self.r) * self.mj

    def vj(self, v):
        return v[self.j] * (~self.wall)[..., None]

    def density(self):
        self.rho = self.m / (math.pi * self.h ** 3) + (self.mj * self.W(self.r)).sum(1)

    def alpha_(self):
        a1 = (self.xij * self.fm[..., None]).sum(1)
        a2 = ((self.fm * self.r) ** 2 * ~self.wall).sum(1)
        self.alpha = self.rho / ((a1 * a1).sum(1) + a2).clamp(min=1e-6)

    def div(self, v):
        return (self.fm * (self.xij * (v[:, None] - self.vj(v))).sum(2)).sum(1)

    def push(self, v, k, dt):
        kk = k[:, None] + k[self.j] * ~self.wall
        return v - dt * (self.xij * (self.fm * kk)[..., None]).sum(1)

    def approach(self):
        return (self.xij * (self.v[:, None] - self.vj(self.v))).sum(2).clamp(max=0)

    def wcsph(self, steps, kw):
        f = lambda k: float(np.float32(kw[k]))  # noqa: E731
        dt, cs, hs, gam = f("dt"), f("soundSpeed_cs"), 2 * self.h, f("wc_gamma")
        visc, bvisc = float(np.float32(VISC)), f("boundary_visc")
        for _ in range(steps):
            self.search()
            self.density()
            p = (self.rho0 * cs * cs / gam * ((self.rho / self.rho0) ** gam - 1)).clamp(min=0)
            own = (p / self.rho ** 2)[:, None]
            rj = torch.where(self.wall, self.rho[:, None].expand_as(self.r), self.rho[self.j])
            press = own + torch.where(self.wall, own.expand_as(self.r), (p / self.rho ** 2)[self.j])
            nu = 2 * torch.where(self.wall, torch.full_like(self.r, bvisc), torch.full_like(self.r, visc)) * hs * cs
            pi = -nu / (self.rho[:, None] + rj) * self.approach() / (self.r ** 2 + 0.01 * hs * hs)
            a = self.g + (self.xij * (-self.fm * (press + pi))[..., None]).sum(1)
            self.v = self.v + a * dt
            self.x = self.x + self.v * dt

    def dfsph(self, steps, kw):
        hs, nu = 2 * self.h, float(np.float32(kw["nu"]))
        self.search()
        self.density()
        self.alpha_()
        for _ in range(steps):
            dt = float(np.float32(kw["cfl_factor"])) * self.d / float(self.v.norm(dim=1).max())
            dt = min(max(dt, float(np.float32(kw["dt_min"]))), float(np.float32(kw["dt_max"])))
            rj = torch.where(self.wall, self.rho[:, None].expand_as(self.r), self.rho[self.j])
            t = 10 * nu * self.fm / rj * self.approach() / (self.r ** 2 + 0.01 * hs * hs)
            v = self.v + dt * (self.g + (self.xij * t[..., None]).sum(1))
            it = 0
            while True:
                adv = (self.rho + dt * self.div(v)).clamp(min=self.rho0)
                err = float(adv.mean()) / self.rho0 - 1
                v = self.push(v, (adv - self.rho0) / dt ** 2 * self.alpha / self.rho, dt)
                it += 1
                if not ((err > kw["df_density_goal"] or it < kw["df_density_min_iter"]) and
                        it < kw["df_density_max_iter"]):
                    break
            self.x = self.x + v * dt
            self.search()
            self.density()
            self.alpha_()
            it = 0
            while True:
                dd = self.div(v)
                dd = torch.where((dd < 0) | (self.rho + dd * dt < self.rho0), torch.zeros_like(dd), dd)
                err = float(dd.mean()) * dt / self.rho0
                v = self.push(v, dd * self.alpha / dt / self.rho, dt)
                it += 1
                if not ((err > kw["df_div_goal_rel"] or it < kw["df_div_min_iter"]) and it <= kw["df_div_max_iter"]):
                    break
            self.v = v


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        scs = _batch_scenes(case, seed)
    elif kind in ("wcsph", "dfsph", "dfsph_host"):
        scs = [_scene(case, seed)]
    else:
        return None
    x, v = [], []
    for sc in scs:
        e = _Exact(sc)
        if kind == "wcsph":
            e.wcsph(case["steps"], WCSPH_KW)
        else:
            e.dfsph(case["steps"], DFSPH_KW)
        x.append(e.x.cpu())
        v.append(e.v.cpu())
    out = {"position": torch.cat(x), "velocity": torch.cat(v)}
    return out if kind == "dfsph_host" else {**out, "n_fluid": None}
