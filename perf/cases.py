"""The work whose speed this package is judged by: calls of its public entry
points on fluid scenes from a few hundred to 1.4 million particles.

Each case is one of these kinds (`kind`):

* `frames`   -- an episode of the plugin classes: `Framework.reset()` (particles
                back to their start, lists rebuilt) and `frames` times
                `Framework.forward()`, as an interactive program does, or one
                `Framework.forward_many(frames)` with `queued`;
* `batch`    -- several independent scenes in one `Engine`, restarted, built and
                stepped `frames` times: the batched form;
* `hosted`   -- one step of a program that keeps x and v in host memory: upload
                of the positions, `Engine.build`, `Engine.step_io`, statistics;
* `build`    -- `NeighbourSearch.build_cache`: lists, density and k;
* `ip`, `prj`, `viscosity`, `tension` -- one solver on its own over lists that
                are there already: `IP.solve`, `PRJ.solve`, and the engine's two
                implicit non-pressure solves;
* `density`  -- `ivp_density_aii_noalloc`, the entry point without a workspace.

The particle states are those of a scene that has been running: fluid at rest
density (a lattice of 0.93 of the particle spacing with 15 % jitter: about 34
neighbours at irregular distances, and one to three outer updates a solve, as in
a collapse under way), a spreading column's velocity field with noise, and one
layer of wall particles in the reference's layout.  Everything comes from the
seed, so both sides of a comparison step the same particles.
"""
import ctypes
import math

import numpy as np
import torch

from implicitvelocityprojection_b200 import _lib
from implicitvelocityprojection_b200 import scenes as S
from implicitvelocityprojection_b200.config import SimConfig
from implicitvelocityprojection_b200.engine import Engine
from implicitvelocityprojection_b200.framework import Framework
from implicitvelocityprojection_b200.ip import IP
from implicitvelocityprojection_b200.neighbour_search import NeighbourSearch
from implicitvelocityprojection_b200.prj import PRJ
from implicitvelocityprojection_b200.simulation_data import SimulationData

SPACING = 0.02        # particle diameter of the column scenes (m)
SPACING_FINE = 0.01   # of the dam break with surface tension
PACK = 0.93           # lattice step over the diameter: rest density 1000 with m = 0.8 d^3 rho0
NEIGHBOURS = 34       # neighbours of a particle in such a fluid, walls included


def listed():
    return [
        # the smallest thing a user steps: a test block, interactive, where
        # launches and the statistics read count
        dict(name="block_768_frames", kind="frames", n=768, shape="block", frames=4),
        # the small column collapse, IP only, one frame after another
        dict(name="column_8k_frames", kind="frames", n=8192, shape="column", frames=4),
        # the headline scene: the tall column with implicit viscosity,
        # queued as a production run does
        dict(name="column_102k_viscous", kind="frames", n=102400, shape="column", visc=True, frames=2, queued=True),
        # the largest single scene: dam break with viscosity and surface tension
        dict(name="dam_524k_full", kind="frames", n=524288, shape="dam", visc=True, tension=True, frames=1),
        # the batched form: 64 columns of 4,096 to 65,536 particles
        dict(name="batch_64", kind="batch", scenes=64, lo=4096, hi=65536, mix=0, frames=1),
        # a coupled program whose particles live in host memory
        dict(name="column_102k_hosted", kind="hosted", n=102400, shape="column", visc=True),
        # neighbour search with density and k on the largest served scene
        dict(name="build_262k", kind="build", n=262144, shape="dam"),
        # the pressure solvers on their own, at ragged sizes
        dict(name="ip_31k", kind="ip", n=31007, shape="column"),
        dict(name="prj_102k", kind="prj", n=102400, shape="column"),
        # the two implicit forces on their own
        dict(name="viscosity_102k", kind="viscosity", n=102400, shape="column", visc=True),
        dict(name="tension_130k", kind="tension", n=130011, shape="dam", tension=True),
        # density and k for a caller that cannot allocate
        dict(name="density_40k", kind="density", n=40000, shape="column"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frames", "frames", "frames", "batch", "hosted", "build", "ip", "prj", "viscosity", "tension",
                       "density"])
    shape = rng.choice(["column", "dam", "block"])
    if kind == "frames":
        n = log(500, 300000)
        tension = rng.random() < 0.3
        return dict(kind=kind, n=n, shape=shape, visc=rng.random() < 0.5, tension=tension,
                    frames=rng.randint(1, 4) if n < 100000 else 1, queued=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 40), lo=log(1000, 4096), hi=log(8192, 65536),
                    mix=rng.randint(1, 1 << 20), frames=rng.randint(1, 2))
    if kind == "density":
        return dict(kind=kind, n=log(500, 42000), shape=shape)
    c = dict(kind=kind, n=log(2000, 262144), shape=shape)
    if kind == "viscosity" or (kind == "hosted" and rng.random() < 0.5):
        c["visc"] = True
    if kind == "tension":
        c["tension"] = True
    return c


# ------------------------------------------------------------------- scenes

def _counts(n, shape):
    """Lattice counts (x, y, z) of at least n particles, the top layer partly
    filled: a column (square base, height 1.6 of the width), a dam-break block
    (2:1:1) or a flat block (height 0.6 of the width)."""
    rise, long = {"column": (1.6, 1), "dam": (1.0, 2), "block": (0.6, 1)}[shape]
    w = max(2, int(round((n / (rise * long)) ** (1.0 / 3.0))))
    return long * w, max(2, -(-n // (long * w * w))), w


def _scene(n, shape, seed, visc=False, tension=False, **kw):
    rng = np.random.default_rng([seed, n])
    d = SPACING_FINE if tension else SPACING
    counts = _counts(n, shape)
    step, gap, margin = PACK * d, 1.6 * d, 4.0 * d
    lower = [margin + gap] * 3
    ix = np.stack(np.meshgrid(*[np.arange(c) for c in counts], indexing="ij"), -1).reshape(-1, 3)
    order = np.argsort(ix[:, 1], kind="stable")[:n]       # the lowest n, back in lattice order
    ix = ix[np.sort(order)]
    x = np.asarray(lower) + step * (ix + rng.uniform(-0.15, 0.15, size=ix.shape))
    extent = [(c - 1) * step for c in counts]
    # walls: beside the column, tight in depth for the dam break, twice as long
    # as the fluid where it spreads
    free = {"column": (1.0, 1.5, 1.0), "dam": (2.2, 1.6, 1.0), "block": (2.0, 2.0, 2.0)}[shape]
    box = [d * math.ceil((free[a] * extent[a] + 2.0 * gap) / d) for a in range(3)]
    domain = [b + 2.0 * margin for b in box]
    shell = S.cube_shell([margin + 0.5 * b for b in box], box, d, layers=1)
    a = 1.5                                               # spreading rate (1/s)
    u = x - np.asarray(lower) - 0.5 * np.asarray([extent[0], 0.0, extent[2]])
    v = np.stack([0.5 * a * u[:, 0], -a * u[:, 1], 0.5 * a * u[:, 2]], -1) + rng.normal(0.0, 0.02, size=x.shape)
    if visc:
        kw.update(viscosity_method=1, viscosity_coeff=1e-3)
    if tension:
        kw.update(surface_tension_method=1, surface_tension_coeff=0.05, dt=5e-4)
    return S.assemble([x.astype(np.float32)], [shell], particle_radius=0.5 * d, domain_size=domain,
                      fluid_velocity=v.astype(np.float32), name="%s_%d" % (shape, n), **kw)


def _options(case):
    return {k: case[k] for k in ("visc", "tension") if case.get(k)}


def _mix(case):
    """(fluid count, shape) of a batch's scenes, counts log-uniform."""
    rng = np.random.default_rng(case["mix"])
    return [(int(c), "column") for c in
            np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), size=case["scenes"]))]


def _scenes(case, seed):
    if case["kind"] == "batch":
        return [_scene(n, shape, seed + 7919 * i) for i, (n, shape) in enumerate(_mix(case))]
    return [_scene(case["n"], case["shape"], seed, **_options(case))]


# ---------------------------------------------------------------- the cases

def _plugins(sc, method=1):
    sc.pressure_method = method
    cfg = SimConfig.from_scene(sc)
    ps = SimulationData.from_scene(sc, cfg)
    return cfg, ps, NeighbourSearch(ps.domain_size, ps.support_radius, ps)


def prepare(case, seed):
    kind = case["kind"]
    scs = _scenes(case, seed)
    sc = scs[0]
    st = {"case": case}
    if kind == "frames":
        cfg, ps, ns = _plugins(sc)
        st.update(ps=ps, fw=Framework(ps, ns, cfg))
        st["fw"].initialize()
    elif kind in ("build", "ip", "prj"):
        cfg, ps, ns = _plugins(sc, 0 if kind == "prj" else 1)
        solver = (PRJ if kind == "prj" else IP)(ps, ns, cfg)
        ns.build_cache(ps.x, ps.particle_num, ps.cache_size, solver=solver)
        st.update(ps=ps, ns=ns, solver=solver, dt=cfg.dt)
    elif kind == "density":
        m, _ = sc.masses()
        st.update(x=torch.from_numpy(sc.x).cuda(), m=torch.from_numpy(m).cuda(),
                  dynamic=torch.from_numpy(sc.is_dynamic).cuda(), sc=sc,
                  density=torch.from_numpy(sc.density0).cuda(), k=torch.zeros(sc.n, device="cuda"),
                  domain=(ctypes.c_float * 3)(*[float(a) for a in sc.domain_size]), lib=_lib.load())
    else:
        eng = Engine(scs)
        st.update(eng=eng, x0=eng.arrays["x"].clone(), v0=eng.arrays["v"].clone())
        if kind in ("viscosity", "tension"):
            eng.build()
        else:
            eng.prepare()
        if kind == "hosted":
            n = st["n"] = sc.n_dynamic
            st.update({k: torch.from_numpy(a[:n].copy()).pin_memory() for k, a in (("x_in", sc.x), ("v_in", sc.v))})
            st.update({k: torch.empty(n, 3).pin_memory() for k in ("x_out", "v_out")})
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "frames":
        fw, ps = st["fw"], st["ps"]
        fw.reset()
        if case.get("queued"):
            fw.forward_many(case["frames"])
        else:
            for _ in range(case["frames"]):
                fw.forward()
        return {"x": ps.x, "v": ps.v, "density": ps.density, "k": ps.k}
    if kind == "batch":
        eng = st["eng"]
        eng.arrays["x"].copy_(st["x0"])
        eng.arrays["v"].copy_(st["v0"])
        eng.build()
        eng.step(case["frames"])
        return {k: eng.arrays[k] for k in ("x", "v", "density", "k")}
    if kind == "hosted":
        eng, n = st["eng"], st["n"]
        eng.arrays["x"][:n].copy_(st["x_in"], non_blocking=True)
        eng.build()
        eng.step_io(None, st["v_in"], st["x_out"], st["v_out"], first=0, count=n)
        eng.stats(0)                                      # waits for the step, as its reader must
        return {"x": st["x_out"], "v": st["v_out"]}
    if kind == "build":
        ps = st["ps"]
        st["ns"].build_cache(ps.x, ps.particle_num, ps.cache_size, solver=st["solver"])
        return {"density": ps.density, "k": ps.k}
    if kind in ("ip", "prj"):
        ps = st["ps"]
        ps.v.copy_(ps.v0)
        st["solver"].solve(st["dt"])
        return {"v": ps.v, "divergence": ps.divergence}
    if kind in ("viscosity", "tension"):
        eng = st["eng"]
        eng.arrays["v"].copy_(st["v0"])
        eng.viscosity_solve() if kind == "viscosity" else eng.surface_tension_solve()
        return {"v": eng.arrays["v"]}
    p = ctypes.c_void_p
    status = st["lib"].ivp_density_aii_noalloc(
        p(st["x"].data_ptr()), p(st["m"].data_ptr()), p(st["dynamic"].data_ptr()), st["sc"].n,
        ctypes.c_float(st["sc"].particle_radius), ctypes.cast(st["domain"], p), st["sc"].cache_size,
        p(st["density"].data_ptr()), p(st["k"].data_ptr()), p(torch.cuda.current_stream().cuda_stream))
    _lib.check(status, "ivp_density_aii_noalloc")
    return {"density": st["density"], "k": st["k"]}


def work(case):
    """Bytes: the particle arrays a call must read and write, once.  Flops: the
    pair sums it cannot do without, at the fewest solver passes such a state
    takes (a build; one outer update of two CG iterations; two iterations of
    an implicit force; three projected-Jacobi passes)."""
    kind = case["kind"]
    n = sum(c for c, _ in _mix(case)) if kind == "batch" else case["n"]
    pairs = NEIGHBOURS * n
    build = 45.0 * pairs                                  # distance, spline, gradient, density and Aii terms
    ip = pairs * (2 * 9.0 + 9.0 + 2 * (9.0 + 8.0))        # two packs, right-hand side, two times A and B
    visc, ten = pairs * (45.0 + 2 * 22.0), pairs * (9.0 + 60.0 + 2 * 10.0)
    if kind in ("frames", "batch", "hosted"):
        forces = (visc if case.get("visc") else 0.0) + (ten if case.get("tension") else 0.0)
        k = case.get("frames", 1)
        return {"bytes": n * (36.0 + 32.0), "flops": (k + 1) * build + k * (ip + forces)}
    if kind in ("build", "density"):
        return {"bytes": n * (20.0 + 8.0), "flops": build}
    one = {"ip": ip, "prj": 3 * pairs * 17.0, "viscosity": visc, "tension": ten}[kind]
    return {"bytes": n * (12.0 + 12.0 + 16.0 + 4.0), "flops": one}


def tolerance(case):
    # Measured against exact(), times about four.  Build: 1.9e-7 (k).  Forces:
    # 3.6e-8 (v changes little).  PRJ: 2.3e-6.  IP and frames are 1e-6 to 1e-5
    # off as a rule, but a particle whose constraint rho - rho0 + J d lies
    # within its 32-bit rounding of zero may fall on either side of the
    # operator's switch, which changes the velocities beside it: 4e-3 seen on
    # 4,000 particles, 1e-4 on a million.
    kind = case["kind"]
    if kind in ("build", "density"):
        return {"rel": 8e-7, "max": 4e-5}
    if kind in ("viscosity", "tension"):
        return {"rel": 2e-7, "max": 1e-5}
    if kind == "prj":
        return {"rel": 1e-5, "max": 4e-3}
    return {"rel": 5e-3, "max": 0.99}


# ------------------------------------------------- the same in 64 bits

def _pairs(x, dyn, h):
    """(i, j) of every dynamic i and every j != i with |x_i - x_j| < h."""
    dev = x.device
    lo = x.min(0).values
    cell = ((x - lo) / h).floor().long() + 1
    dims = cell.max(0).values + 2
    key = (cell[:, 2] * dims[1] + cell[:, 1]) * dims[0] + cell[:, 0]
    order = torch.argsort(key)
    start = torch.searchsorted(key[order], torch.arange(int(dims.prod()) + 1, device=dev))
    mine = torch.nonzero(dyn).flatten()
    found_i, found_j = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            at = key[mine] + (dz * dims[1] + dy) * dims[0]
            b, e = start[at - 1], start[at + 2]
            count = e - b
            i = torch.repeat_interleave(mine, count)
            off = torch.arange(int(count.sum()), device=dev) - torch.repeat_interleave(count.cumsum(0) - count, count)
            j = order[torch.repeat_interleave(b, count) + off]
            near = ((x[i] - x[j]).square().sum(1) < h * h) & (i != j)
            found_i.append(i[near])
            found_j.append(j[near])
    return torch.cat(found_i), torch.cat(found_j)


class _Exact:
    """One scene in 64 bits, with the reference's formulas and stopping rules."""

    def __init__(self, sc, device):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device).double()  # noqa: E731
        f = lambda a: float(np.float32(a))  # noqa: E731
        self.sc = sc
        self.x, self.v, self.m, self.rho0 = t(sc.x), t(sc.v), t(sc.masses()[0]), t(sc.density0)
        self.dyn = t(sc.is_dynamic) == 1
        self.fluid = self.dyn & (t(sc.material) == 1)
        self.d, self.dt = f(sc.particle_diameter), f(sc.dt)
        self.h = 2.0 * self.d
        self.gravity = torch.tensor([f(g) for g in sc.gravity], dtype=torch.float64, device=device)
        self.domain = t(sc.domain_size)
        self.density, self.k = self.rho0.clone(), torch.zeros_like(self.m)

    def sum(self, values):
        out = torch.zeros((self.x.shape[0],) + values.shape[1:], dtype=torch.float64, device=self.x.device)
        return out.index_add_(0, self.i, values)

    def mean(self, values):
        return float(values[self.dyn].clamp(min=0.0).sum()) / max(int(self.dyn.sum()), 1)

    def cubic(self, r, h):
        q = r / h
        return 8.0 / math.pi / h ** 3 * torch.where(
            q <= 0.5, 6.0 * (q ** 3 - q ** 2) + 1.0, 2.0 * (1.0 - q).clamp(min=0.0) ** 3)

    def build(self):
        h = self.h
        self.i, self.j = _pairs(self.x, self.dyn, h)
        self.xij = self.x[self.i] - self.x[self.j]
        self.r = self.xij.norm(dim=1)
        rc = self.r.clamp(min=1e-6)
        mj = self.m[self.j]
        self.J = (-mj * 45.0 / (math.pi * h ** 6) * (h - rc) ** 2 / rc)[:, None] * self.xij
        rho = self.m * 8.0 / math.pi / h ** 3 + self.sum(mj * self.cubic(self.r, h))
        aii = self.sum(torch.where(self.dyn[self.j], self.J.square().sum(1) / mj, 0.0))
        aii = aii + self.sum(-self.J).square().sum(1) / self.m
        self.density = torch.where(self.dyn, rho, self.density)
        self.k = torch.where(self.dyn, 1.0 / (aii + 1e-3), 0.0)

    def div(self, u):
        return self.sum(((u[self.i] - u[self.j]) * self.J).sum(1))

    def grad(self, y):
        w = y / self.m
        return self.sum((y[self.i] + self.m[self.i] * w[self.j])[:, None] * self.J)

    def ip(self):
        sc, dyn3 = self.sc, self.dyn[:, None]
        c = self.density - self.rho0
        d = torch.where(dyn3, self.dt * self.v, 0.0)
        updates = 0
        while True:
            t = torch.where(self.dyn, self.div(d) + c, 0.0)
            f = t.clamp(min=0.0)
            err = self.mean(f / self.rho0)
            if (err < sc.density_error_tol and updates >= 1) or updates >= sc.max_outer_iters:
                break
            s = torch.where(t >= 1e-6, self.k, 0.0)
            r = sc.omega * self.grad(f * self.k)
            sol, p, rr, it = torch.zeros_like(d), r.clone(), float(r.square().sum()), 0
            while rr > 1e-30:
                ap = torch.where(dyn3, self.m[:, None] * p + sc.omega * self.grad(s * self.div(p)), 0.0)
                alpha = rr / max(float((p * ap).sum()), 1e-30)
                sol, r = sol + alpha * p, r - alpha * ap
                new, it = float(r.square().sum()), it + 1
                if (new < sc.tol_pcg and it >= 2) or it >= sc.max_iteration_pcg:
                    break
                p, rr = r + new / max(rr, 1e-30) * p, new
            d = d - sol
            updates += 1
        self.finish(d)

    def prj(self):
        sc, dyn3 = self.sc, self.dyn[:, None]
        c = self.density - self.rho0
        start = torch.where(dyn3, self.dt * self.v, 0.0)
        lam, updates = torch.zeros_like(c), 0
        while True:
            d = torch.where(dyn3, start - self.grad(lam) / self.m.clamp(min=1e-6)[:, None], 0.0)
            r = torch.where(self.dyn, self.div(d) + c, 0.0)
            lam = (lam + 0.5 * r * self.k).clamp(min=0.0)
            err = self.mean(r / self.rho0)
            if (err < sc.density_error_tol and updates >= 1) or updates >= sc.max_outer_iters:
                break
            updates += 1
        self.finish(d)

    def finish(self, d):
        self.divergence = torch.where(self.dyn, self.div(d / self.dt).clamp(min=0.0), 0.0)
        self.v = torch.where(self.dyn[:, None], d / self.dt, self.v)

    def cg(self, apply, solve, rhs, cap):
        """The preconditioned CG of the two implicit forces (tolerance 1e-5)."""
        x, r = torch.zeros_like(rhs), rhs
        z = solve(r)
        p, rz, it = z, float((r * z).sum()), 0
        while rz > 1e-12 or it:
            ap = apply(p)
            pap = float((p * ap).sum())
            if pap <= 0.0:
                break
            alpha = rz / max(pap, 1e-12)
            x, r, it = x + alpha * p, r - alpha * ap, it + 1
            z = solve(r)
            if (float(r.square().sum()) < 1e-5 and it >= 2) or it >= cap:
                break
            new = float((r * z).sum())
            p, rz = z + new / max(rz, 1e-12) * p, new
        return x

    def viscosity(self):
        i, j, fl = self.i, self.j, self.fluid
        c = torch.where(fl[j] & fl[i], 10.0 / self.density[j], 0.0) / (self.r ** 2 + 0.01 * self.h ** 2)
        f = float(np.float32(self.sc.viscosity_coeff)) * self.dt * self.rho0 / self.density
        m = torch.eye(3, dtype=torch.float64, device=self.x.device) - f[:, None, None] * self.sum(
            c[:, None, None] * self.J[:, :, None] * self.xij[:, None, :])
        inv = torch.linalg.inv(m)
        lap = lambda u: f[:, None] * self.sum(  # noqa: E731
            (c * ((u[i] - u[j]) * self.xij).sum(1))[:, None] * self.J)
        dyn3 = self.dyn[:, None]
        v = torch.where(dyn3, self.v, 0.0)
        self.v = self.v + self.cg(lambda p: p - lap(p), lambda r: (inv @ r[:, :, None])[:, :, 0], lap(v), 1000)

    def tension(self):
        i, j, dt, hs = self.i, self.j, self.dt, self.h
        sigma, d = float(np.float32(self.sc.surface_tension_coeff)), self.d
        on = self.fluid[i] & self.fluid[j]
        v = self.v
        vij = v[i] - v[j]
        div = self.sum(torch.where(on, (vij * self.J).sum(1), 0.0))
        rbar = 0.5 * (self.density[i] + self.density[j])
        theta, q = 10.0 / 7.0, self.r / hs
        w = theta * self.cubic(self.r.clamp(min=d), hs)
        slope = torch.where(q <= 0.5, -12.0 * q + 18.0 * q * q, -6.0 * (1.0 - q) ** 2)
        slope = torch.where(self.r > d, theta * 8.0 / (math.pi * hs ** 4) * slope, 0.0)
        gv = slope * (self.xij * vij).sum(1) / self.r.clamp(min=1e-12)
        g = w / rbar + dt * (gv / rbar - w / (2.0 * rbar * rbar) * (div[i] + div[j]))
        g = torch.where(on, g, 0.0) * 0.5 * (self.m[i] + self.m[j])
        f = torch.where(self.fluid, dt * dt * sigma / self.m, 0.0)
        push = torch.where(self.fluid, -dt * sigma / self.m, 0.0)[:, None] * self.sum(g[:, None] * self.xij)
        spread = lambda u: f[:, None] * self.sum(g[:, None] * (u[i] - u[j]))  # noqa: E731
        inv = 1.0 / (1.0 + f * self.sum(g)).clamp(min=1e-12)
        self.v = v + self.cg(lambda p: p + spread(p), lambda r: inv[:, None] * r, push - spread(v), 100)

    def advect(self):
        dyn3 = self.dyn[:, None]
        v = torch.where(dyn3, self.v, 0.0)
        x = self.x + self.dt * v
        high, low = x > self.domain - self.h, x <= self.h
        n = torch.where(dyn3, high.double() - low.double(), 0.0)
        at = torch.minimum(torch.maximum(x, torch.full_like(self.domain, self.h)), self.domain - self.h)
        self.x = torch.where(dyn3, at, x)
        n = n / n.norm(dim=1, keepdim=True).clamp(min=1e-6)
        self.v = v - 1.5 * (v * n).sum(1, keepdim=True) * n

    def frame(self):
        self.v = self.v + torch.where(self.dyn[:, None], self.gravity * self.dt, 0.0)
        if self.sc.surface_tension_method:
            self.tension()
        if self.sc.viscosity_method:
            self.viscosity()
        self.ip()
        self.advect()
        self.build()


def exact(case, seed):
    kind = case["kind"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    outs = []
    for sc in _scenes(case, seed):
        e = _Exact(sc, device)
        e.build()
        if kind in ("frames", "batch", "hosted"):
            for _ in range(case.get("frames", 1)):
                e.frame()
        elif kind in ("ip", "prj", "viscosity", "tension"):
            getattr(e, kind)()
        outs.append(e)
        if kind != "frames" and kind != "batch":
            break
    names = {"frames": ("x", "v", "density", "k"), "batch": ("x", "v", "density", "k"), "hosted": ("x", "v"),
             "build": ("density", "k"), "density": ("density", "k"), "ip": ("v", "divergence"),
             "prj": ("v", "divergence")}.get(kind, ("v",))
    got = {k: torch.cat([getattr(e, k) for e in outs]) for k in names}
    if kind == "hosted":
        got = {k: a[outs[0].dyn] for k, a in got.items()}
    return got
