"""Performance cases: one advection step of every solver, over the sizes it is used at.

A pass is one advection step through the public entry points, started from a given state:
the state is loaded (device copies, ``sphx_mp_upload`` or ``sphx_mp_upload_host``), the
configuration of that state is built and the step's relaxation runs.  That is the work of
one step of a driver's main loop with the configuration update first instead of last, so
every pass of a case does the same work and no pass depends on the one before it.  The
batched solver has no load: its passes are two steps each and follow one another.

The states are moderately disordered flows: the lattice of the case moved by a smooth
area-preserving displacement of up to a few spacings plus a small random jitter, a swirling
velocity field and the left-over force and density rate of an earlier step.

The mixed-precision solver holds velocity, density and pressure in FP32; those outputs are
returned in FP32 (positions, which it integrates in FP64, in FP64).
"""
import math

import numpy as np
import torch

from sphinxsys_gb300 import cases as C
from sphinxsys_gb300 import native as N
from sphinxsys_gb300 import sph as S
from sphinxsys_gb300.batch import BatchDamBreak
from sphinxsys_gb300.dambreak import DamBreak, DamBreakCKNested, MixedPrecisionDamBreak
from sphinxsys_gb300.taylor_green import MixedPrecisionTaylorGreen, TaylorGreen

DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # Dambreak.cpp as the reference ships it: a few thousand particles, every call latency bound
        {"name": "fp64 2d dp 0.025", "kind": "fp64", "dim": 2, "dp": 0.025},
        # the reference's 3D dam break with its six wall probes read every step
        {"name": "fp64 3d reference tank dp 0.05", "kind": "probes", "dim": 3, "dp": 0.05},
        # a production FP64 run: 1,702,400 particles
        {"name": "fp64 3d dp 0.0075", "kind": "fp64", "dim": 3, "dp": 0.0075},
        # the SYCL driver's particle methods (tabulated kernel, correction matrices), 90,000 particles
        {"name": "ck 3d dp 0.02", "kind": "ck", "dim": 3, "dp": 0.02},
        # mixed precision: a 2D study
        {"name": "mixed 2d dp 0.005", "kind": "mixed", "dim": 2, "dp": 0.005},
        # mixed precision: a coarse 3D run, where launches and latency count
        {"name": "mixed 3d dp 0.03", "kind": "mixed", "dim": 3, "dp": 0.03},
        # mixed precision: the headline tank, 3,340,000 particles
        {"name": "mixed 3d dp 0.006", "kind": "mixed", "dim": 3, "dp": 0.006},
        # mixed precision coupled to a host program: FP64 rows in and out every step
        {"name": "mixed host rows 3d dp 0.01", "kind": "rows", "dim": 3, "dp": 0.01},
        # parameter studies: independent instances advanced together, results read back
        {"name": "batch 2d 8 x 50000", "kind": "batch", "dim": 2, "count": 8, "n": 50000, "steps": 2},
        {"name": "batch 3d 8 x 40000", "kind": "batch", "dim": 3, "count": 8, "n": 40000, "steps": 2},
        # periodic flows: the 3D vortex in mixed precision, the reference's 2D vortex in FP64
        {"name": "taylor-green mixed 3d 128", "kind": "tg-mixed", "dim": 3, "resolution": 128},
        {"name": "taylor-green fp64 2d 100", "kind": "tg-fp64", "dim": 2, "resolution": 100},
    ]


def draw(rng):
    def spread(lo, hi):
        return float(round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 6))

    kind = rng.choice(["fp64", "fp64", "probes", "ck", "mixed", "mixed", "rows", "batch", "tg-mixed", "tg-fp64"])
    dim = rng.choice([2, 3])
    if kind == "probes":
        return {"kind": kind, "dim": 3, "dp": spread(0.02, 0.06)}
    if kind == "fp64":
        return {"kind": kind, "dim": dim, "dp": spread(0.004, 0.03) if dim == 2 else spread(0.009, 0.05)}
    if kind == "ck":
        return {"kind": kind, "dim": dim, "dp": spread(0.006, 0.03) if dim == 2 else spread(0.016, 0.05)}
    if kind == "mixed":
        return {"kind": kind, "dim": dim, "dp": spread(0.002, 0.02) if dim == 2 else spread(0.0075, 0.04)}
    if kind == "rows":
        return {"kind": kind, "dim": dim, "dp": spread(0.002, 0.02) if dim == 2 else spread(0.009, 0.03)}
    if kind == "batch":
        return {"kind": kind, "dim": dim, "count": rng.randint(3, 10), "n": int(spread(20000, 60000)), "steps": 2}
    if kind == "tg-mixed":
        return {"kind": kind, "dim": dim, "resolution": int(spread(100, 700) if dim == 2 else spread(32, 127))}
    return {"kind": kind, "dim": dim, "resolution": int(spread(40, 300) if dim == 2 else spread(20, 72))}


# ------------------------------------------------------------------ inputs
def tank(case):
    if case["kind"] == "probes":
        t = C.dambreak_3d_reference(case["dp"])
        # the reference's probe heights, on the wetted wall
        t.observers = [(0.0, y, z) for (_, y, z) in t.observers]
        return t
    return C.dambreak_2d(case["dp"]) if case["dim"] == 2 else C.dambreak_3d(case["dp"])


def instances(case, seed):
    """Water columns of about n particles each, H = 1, aspects spread over [0.25, 1], in
    tanks of the dam-break ratios; the gravity of each is drawn from the seed."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["count"]):
        L, dim = 1.0 / (0.25 + 0.75 * ((0.37 + 0.618034 * k) % 1.0)), case["dim"]
        gravity = rng.uniform(0.8, 1.25)
        size = [L, 1.0] if dim == 2 else [L, 0.5 * L, 1.0]
        box = [2.683 * L, 5.366] if dim == 2 else [2.683 * L, 0.5 * L, 5.366]
        dp = (math.prod(size) / case["n"]) ** (1.0 / dim)
        pad = [0.0] * (3 - dim)
        lo, up = [-4 * dp] * dim, [b + 4 * dp for b in box]
        water, inner = [0.5 * s for s in size], [0.5 * b for b in box]
        g = [0.0] * dim
        g[-1] = -gravity
        out.append(C.DamBreakCase(
            name="column%d" % k, dim=dim, sys_lower=tuple(lo + pad), sys_upper=tuple(up + pad), dp=dp,
            water_center=tuple(water + pad), water_halfsize=tuple(water + pad), outer_center=tuple(inner + pad),
            outer_halfsize=tuple([b + 4 * dp for b in inner] + pad), inner_center=tuple(inner + pad),
            inner_halfsize=tuple(inner + pad), rho0=1.0, c0=20.0 * math.sqrt(gravity),
            U_ref=2.0 * math.sqrt(gravity), gravity=tuple(g + pad),
            observers=[], loop_style=0, vertical_axis=dim - 1))
    return out


def lattice(t, part):
    """Lattice points (n x dim, host) of the water block or the tank wall of a case, in the
    generator's order."""
    d, dp = t.dim, t.dp
    axes = [(t.sys_lower[a] + np.arange(math.ceil((t.sys_upper[a] - t.sys_lower[a]) / dp)) * dp) + 0.5 * dp
            for a in range(d)]

    def box(centre, half):
        m = [np.abs(axes[a] - centre[a]) <= half[a] for a in range(d)]
        return np.ix_(*m), m

    grid = np.zeros([len(a) for a in axes], dtype=bool)
    if part == "water":
        grid[box(t.water_center, t.water_halfsize)[0]] = True
    else:
        grid[box(t.outer_center, t.outer_halfsize)[0]] = True
        grid[box(t.inner_center, t.inner_halfsize)[0]] = False
    at = np.nonzero(grid)
    return np.stack([axes[a][at[a]] for a in range(d)], axis=1)


def disordered(x, lower, size, dp, speed, mass, seed):
    """The state (dim x n, FP64) of a flow in the block [lower, lower + size] whose lattice
    is x (n x dim): position, velocity, force, density, density rate."""
    gen = torch.Generator(DEV).manual_seed(seed)
    host = np.random.default_rng(seed)
    x = torch.from_numpy(np.ascontiguousarray(x.T)).to(DEV)
    d, n = x.shape
    s = [(x[a] - lower[a]) / size[a] for a in range(d)]
    shift, v = torch.zeros_like(x), torch.zeros_like(x)
    up = d - 1  # swirls in the planes of the last axis and each other one
    for a in range(d - 1):
        k1, k2 = int(host.integers(1, 4)), int(host.integers(1, 4))
        sx, cx = torch.sin(math.pi * k1 * s[a]), torch.cos(math.pi * k1 * s[a])
        sz, cz = torch.sin(math.pi * k2 * s[up]), torch.cos(math.pi * k2 * s[up])
        p, q = sx * cz * k2 / size[up], -cx * sz * k1 / size[a]
        scale = 1.0 / max(k2 / size[up], k1 / size[a])
        # a few spacings at most, and small strains where the block is only some spacings wide
        move = min(2.0 * dp, 0.03 * min(size[a] / k1, size[up] / k2)) * host.uniform(0.5, 1.0) * host.choice([-1.0, 1.0])
        flow = speed * host.uniform(0.5, 1.0)
        shift[a] += move * scale * p
        shift[up] += move * scale * q
        v[a] += flow * scale * p
        v[up] += flow * scale * q

    def noise(*shape):
        return 2.0 * torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64) - 1.0

    return {"Position": x + shift + 0.02 * dp * noise(d, n), "Velocity": v + 0.01 * speed * noise(d, n),
            "Force": 0.05 * mass * noise(d, n), "Density": 1.0 + 1e-3 * noise(1, n)[0],
            "DensityChangeRate": 0.05 * noise(1, n)[0]}


def flow(t, seed):
    """A disordered state of the water column of a dam break."""
    lower = [t.water_center[a] - t.water_halfsize[a] for a in range(t.dim)]
    return disordered(lattice(t, "water"), lower, [2 * h for h in t.water_halfsize[:t.dim]], t.dp, 0.5,
                      t.rho0 * t.dp ** t.dim, seed)


def vortex_case(case):
    return C.taylor_green_2d(case["resolution"]) if case["dim"] == 2 else C.taylor_green_3d(case["resolution"])


def vortex(t, seed):
    """A disordered state of a periodic box: jittered lattice, a vortex of random phase."""
    d, m = t.dim, int(math.ceil(t.L / t.dp))
    a = np.arange(m) * t.dp + 0.5 * t.dp
    x = np.stack([g.ravel() for g in np.meshgrid(*[a] * d, indexing="ij")], axis=1)
    st = disordered(x, [0.0] * d, [t.L] * d, t.dp, 0.2 * t.U, t.rho0 * t.dp ** d, seed)
    ph = np.random.default_rng(seed).uniform(0, 2 * math.pi, 2)
    k = 2 * math.pi / t.L
    q = st["Position"]
    st["Velocity"][0] += -t.U * torch.cos(k * q[0] + ph[0]) * torch.sin(k * q[1] + ph[1])
    st["Velocity"][1] += t.U * torch.sin(k * q[0] + ph[0]) * torch.cos(k * q[1] + ph[1])
    st["Position"] = torch.remainder(q, t.L)
    st["Force"].zero_()
    return st


# ------------------------------------------------------------------ device views
class _Array:
    def __init__(self, ptr, shape, dtype):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": dtype, "version": 3}


def view(body, name, ncomp, dtype="<f8"):
    """A body variable (SoA on the device) as a tensor of its own memory."""
    shape = (body.n,) if ncomp == 1 else (ncomp, body.n)
    return torch.as_tensor(_Array(body.device_ptr(name), shape, dtype), device=DEV)


def stream_of(ctx):
    return torch.cuda.ExternalStream(ctx.stream())


def body_like(sim_body):
    """Another body of the same particles, to be written by the solver."""
    body = S.FluidBody(sim_body.system, sim_body.shape, name="Result")
    body.defineMatterMaterial(sim_body.material)
    body._create(sim_body.n)
    for name, nc in (("Position", sim_body.dim), ("Velocity", sim_body.dim), ("Force", sim_body.dim), ("Density", 1),
                     ("Pressure", 1), ("DensityChangeRate", 1)):
        N.call("sphx_body_register", body.handle, name.encode(), N.F64, nc)
    return body


class Loader:
    """Loads a kept state into the variables of a body on the library's stream."""

    def __init__(self, body, state, zero=()):
        self.pairs = [(view(body, k, v.shape[0] if v.dim() == 2 else 1, "<i4" if v.dtype == torch.int32 else "<f8"), v)
                      for k, v in state.items()]
        self.zero = [view(body, k, nc) for k, nc in zero]
        self.stream = stream_of(body.system.ctx)
        torch.cuda.synchronize()
        self()
        body.system.ctx.synchronize()

    def __call__(self):
        with torch.cuda.stream(self.stream):
            for dst, src in self.pairs:
                dst.copy_(src)
            for dst in self.zero:
                dst.zero_()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"kind": kind, "sim": BatchDamBreak(instances(case, seed)), "steps": case["steps"]}
    if kind in ("tg-mixed", "tg-fp64"):
        t = vortex_case(case)
        mixed = kind == "tg-mixed"
        sim = MixedPrecisionTaylorGreen(t) if mixed else TaylorGreen(t)
        body = sim.water_block
        zero = [("ForcePrior", t.dim)]
        if not mixed:
            sim.viscous_force.exec()  # registers its variables
            zero.append(("PreviousViscousForce", t.dim))
        st = {"kind": kind, "sim": sim, "load": Loader(body, vortex(t, seed), zero)}
        if mixed:
            st["out"] = body_like(body)
            st["views"] = solver_views(st["out"])
        else:
            st["views"] = body_views(body)
        return st
    t = tank(case)
    state = flow(t, seed)
    if kind in ("fp64", "probes"):
        sim = DamBreak(t)
        return {"kind": kind, "sim": sim, "load": Loader(sim.water_block, state), "views": body_views(sim.water_block)}
    if kind == "ck":
        sim = DamBreakCKNested(t)
        body, d = sim.water_block, t.dim
        sim.regularization.exec()
        sim.indication.exec()
        state.pop("DensityChangeRate")
        state["CompressionRate"] = 0.05 * torch.sin(37.0 * state["Position"][0])
        state["PreviousSurfaceIndicator"] = torch.ones(body.n, dtype=torch.int32, device=DEV)
        load = Loader(body, state)
        views = {"position": view(body, "Position", d), "velocity": view(body, "Velocity", d),
                 "density": view(body, "Density", 1), "pressure": view(body, "Pressure", 1),
                 "force": view(body, "Force", d), "rate": view(body, "CompressionRate", 1),
                 "correction": view(body, "LinearCorrectionMatrix", d * d), "indicator": view(body, "Indicator", 1, "<i4")}
        return {"kind": kind, "sim": sim, "load": load, "views": views}
    sim = MixedPrecisionDamBreak(t)
    body, d = sim.fp64.water_block, t.dim
    if kind == "mixed":
        load = Loader(body, state)
        out = body_like(body)
        return {"kind": kind, "sim": sim, "load": load, "out": out, "views": solver_views(out)}

    def pinned(a):
        return a.t().contiguous().cpu().pin_memory() if a.dim() == 2 else a.cpu().pin_memory()

    rows = [pinned(state[k]) for k in ("Position", "Velocity", "Force", "Density", "DensityChangeRate")]
    n = body.n
    res = [torch.zeros(s, dtype=torch.float64).pin_memory() for s in ((n, d), (n, d), (n,), (n,))]
    sim.set_host_rows(*[r.numpy() for r in res])
    return {"kind": kind, "sim": sim, "rows": [r.numpy() for r in rows], "keep": rows, "res": res}


def body_views(body):
    d = body.dim
    return {"position": view(body, "Position", d), "velocity": view(body, "Velocity", d),
            "density": view(body, "Density", 1), "pressure": view(body, "Pressure", 1), "force": view(body, "Force", d),
            "rate": view(body, "DensityChangeRate", 1)}


def solver_views(body):
    d = body.dim
    return {"position": view(body, "Position", d), "velocity": view(body, "Velocity", d),
            "density": view(body, "Density", 1), "pressure": view(body, "Pressure", 1)}


# ------------------------------------------------------------------ one pass
def run(state):
    kind, sim = state["kind"], state["sim"]
    if kind == "batch":
        for _ in range(state["steps"]):
            sim.advection_step()
        out = {}
        for q in range(sim.count):
            x, v, rho, p = sim.download(q)
            out["%02d" % q] = [x] + [torch.from_numpy(a).float() for a in (v, rho, p)]
        return out
    if kind == "rows":
        sim.upload_host(*state["rows"])
        sim.advection_step()
        x, v, rho, p = state["res"]
        return {"position": x, "velocity": v.float(), "density": rho.float(), "pressure": p.float()}
    if kind in ("mixed", "tg-mixed"):
        body = sim.fp64.water_block if kind == "mixed" else sim.water_block
        N.call("sphx_mp_upload", sim.handle, body.handle)
        sim.advection_step()
        N.call("sphx_mp_download", sim.handle, state["out"].handle)
        w = state["views"]
        with torch.cuda.stream(state["load"].stream):
            return {"position": w["position"], "velocity": w["velocity"].float(), "density": w["density"].float(),
                    "pressure": w["pressure"].float()}
    state["load"]()
    if kind == "tg-fp64":
        for p in sim.periodic:
            p.bounding_.exec()
        sim.water_block.updateCellLinkedList()
        for p in sim.periodic:
            p.update_cell_linked_list_.exec()
        sim.water_block_inner.updateConfiguration()
        Dt = sim.advection_time_step.exec()
        sim.update_density_by_summation.exec()
        sim.viscous_force.exec()
        sim.transport_velocity_correction.exec()
        t = 0.0
        while t < Dt:
            dt = min(sim.acoustic_time_step.exec(), Dt)
            t += dt
            sim.pressure_relaxation.exec(dt)
            sim.density_relaxation.exec(dt)
        return dict(state["views"], steps=Dt)
    if kind == "ck":
        f64 = sim.fp64
        sim.water_block.updateCellLinkedList()
        f64.water_block_inner.updateConfiguration()
        f64.water_wall_contact.updateConfiguration()
        sim.regularization.exec()
        sim.setup.exec()
        Dt = sim.advection_dt.exec()
        sim.indication.exec()
        sim.correction.exec()
        t = 0.0
        while t < Dt:
            dt = sim.acoustic_dt.exec()
            sim.first_half.exec(dt)
            sim.second_half.exec(dt)
            t += dt
        sim.update_position.exec()
        return dict(state["views"], steps=Dt)
    # classic FP64 dam break
    sim.update_configuration()
    sim.acoustic_dt = 0.0
    _, Dt = sim.relax()
    out = dict(state["views"], steps=Dt)
    if kind == "probes":
        out["probes"] = sim.recorded_pressure.exec()
        out["energy"] = sim.mechanical_energy.exec()
    return out


# ------------------------------------------------------------------ work of one pass
def work(case):
    """Per particle and sweep: its state read and written once (position, velocity, force,
    density, density rate, pressure); two sweeps per acoustic sub-step, five sub-steps per
    advection step, and one configuration.  About 30 operations per pair of a sweep and of
    the configuration.  FP64 state for the FP64 solvers, FP32 for the mixed ones."""
    d, kind = case["dim"], case["kind"]
    if "resolution" in case:
        n = case["resolution"] ** d
    elif kind == "batch":
        n = case["count"] * case["n"]
    else:
        t = tank(case)
        n = math.prod(2 * h / t.dp for h in t.water_halfsize[:d])
    pairs = {2: 20.0, 3: 78.0}[d]
    wide = 8 if kind in ("fp64", "probes", "ck", "tg-fp64") else 4
    sweeps = 11 * case.get("steps", 1)
    host = n * (5 * d + 4) * 8 if kind == "rows" else n * (2 * d + 2) * 8 * (kind == "batch")
    return {"bytes": n * 2 * (3 * d + 3) * wide * sweeps + host, "flops": n * pairs * 30.0 * sweeps}


# ------------------------------------------------------------------ 64-bit reference
def pairs(xi, xj, rc, same):
    """All (i, j) with |x_i - x_j| < rc (dim x n FP64 tensors), i != j when same: i, j, the
    differences (dim rows) and the distance."""
    d = xi.shape[0]
    lo = torch.minimum(xi.min(1).values, xj.min(1).values) - rc
    ci = torch.floor((xi - lo[:, None]) / rc).long()
    cj = torch.floor((xj - lo[:, None]) / rc).long()
    size = [int(max(ci[a].max(), cj[a].max())) + 2 for a in range(d)]

    def key(c):
        k = c[0]
        for a in range(1, d):
            k = k * size[a] + c[a]
        return k

    kj, perm = torch.sort(key(cj))
    found = []
    columns = [(a,) for a in (-1, 0, 1)] if d == 2 else [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)]
    for col in columns:
        c = ci.clone()
        for a, o in enumerate(col):
            c[a] += o
        k = key(c)
        b, e = torch.searchsorted(kj, k - 1), torch.searchsorted(kj, k + 1, right=True)
        cnt = e - b
        for part in torch.arange(xi.shape[1], device=DEV).split(1 << 20):
            m = cnt[part]
            i = torch.repeat_interleave(part, m)
            j = torch.arange(len(i), device=DEV) + torch.repeat_interleave(b[part] - (torch.cumsum(m, 0) - m), m)
            j = perm[j]
            r2 = sum((xi[a][i] - xj[a][j]) ** 2 for a in range(d))
            keep = r2 < rc * rc
            if same:
                keep &= i != j
            found.append((i[keep], j[keep], torch.sqrt(r2[keep])))
    i, j, r = (torch.cat(q) for q in zip(*found))
    return i, j, [xi[a][i] - xj[a][j] for a in range(d)], r


class Kernel:
    """Wendland C2: W and dW/dr; with `tabulated`, the CK form (cubic interpolation in a table)."""

    def __init__(self, dim, h, tabulated=False):
        self.h, self.tabulated = h, tabulated
        self.fW = 7.0 / (4.0 * math.pi * h * h) if dim == 2 else 21.0 / (16.0 * math.pi * h ** 3)
        if tabulated:
            q = (torch.arange(24, device=DEV, dtype=torch.float64) - 1.0) * 0.1
            self.tw, self.tdw = (1.0 - 0.5 * q) ** 4 * (1.0 + 2.0 * q), 0.625 * (q - 2.0) ** 3 * q

    def _cubic(self, table, q):
        loc = torch.floor(q / 0.1)
        i, f1 = loc.long() + 1, q - loc * 0.1
        f0, f2, f3 = f1 + 0.1, f1 - 0.1, f1 - 0.2
        c = 0.1 ** 3
        return (f1 * f2 * f3 / (-6 * c) * table[i - 1] + f0 * f2 * f3 / (2 * c) * table[i]
                + f0 * f1 * f3 / (-2 * c) * table[i + 1] + f0 * f1 * f2 / (6 * c) * table[i + 2])

    def W(self, r):
        q = r / self.h
        return self.fW * (self._cubic(self.tw, q) if self.tabulated else (1.0 - 0.5 * q) ** 4 * (1.0 + 2.0 * q))

    def dW(self, r):
        q = r / self.h
        return self.fW / self.h * (self._cubic(self.tdw, q) if self.tabulated else 0.625 * (q - 2.0) ** 3 * q)


def lattice_sum(dim, k, dp):
    m = int(2 * k.h / dp) + 1
    a = np.arange(-m, m + 1) * dp
    r = np.sqrt(sum(g ** 2 for g in np.meshgrid(*[a] * dim)))
    r = torch.from_numpy(r[r < 2 * k.h])
    q = r / k.h
    return float((k.fW * (1.0 - 0.5 * q) ** 4 * (1.0 + 2.0 * q)).sum())


def onto(n, i, v):
    return torch.zeros(n, device=DEV, dtype=torch.float64).index_add_(0, i, v)


def jump(Z, c0, u):
    """Dissipative pressure jump of the acoustic Riemann solver, limiter slope 3."""
    return Z * u * torch.clamp(3.0 / c0 * torch.clamp(u, min=0.0), max=1.0)


def wall_normals(t, x):
    """Unit normals of wall points (dim x n) from the nearest face of the tank."""
    d = t.dim
    c = torch.tensor(t.inner_center[:d], device=DEV, dtype=torch.float64)[:, None]
    hi = torch.tensor(t.inner_halfsize[:d], device=DEV, dtype=torch.float64)[:, None]
    ho = torch.tensor(t.outer_halfsize[:d], device=DEV, dtype=torch.float64)[:, None]
    p = x - c
    to_inner = torch.maximum(torch.minimum(p, hi), -hi) - p
    gap, axis = (ho - p.abs()).min(0)
    to_outer = torch.zeros_like(p)
    to_outer.scatter_(0, axis[None], (torch.where(torch.gather(p, 0, axis[None]) < 0, -1.0, 1.0) * gap[None]))
    best = torch.where((to_inner.square().sum(0).sqrt() <= gap)[None], to_inner, to_outer)
    return best / best.square().sum(0).sqrt()


class Flow:
    """One fluid, optionally a static wall: the state and the configuration pairs."""

    def __init__(self, dim, dp, c0, gravity, state, t=None):
        self.d, self.dp, self.c0, self.g = dim, dp, c0, gravity
        self.h, self.vol = 1.3 * dp, dp ** dim
        self.m = self.vol  # rho0 = 1
        self.x, self.v, self.F = (state[k].clone() for k in ("Position", "Velocity", "Force"))
        self.rho, self.rate = state["Density"].clone(), state["DensityChangeRate"].clone()
        self.n = self.x.shape[1]
        self.wall = None
        if t is not None:
            w = torch.from_numpy(np.ascontiguousarray(lattice(t, "wall").T)).to(DEV)
            self.wall = w
            self.nw = wall_normals(t, w)

    def configure(self, kernel, period=0.0):
        xj, src = self.x, None
        if period:
            src = torch.arange(self.n, device=DEV)
            for a in range(self.d):
                lo, hi = xj[a] < 2.05 * self.h, xj[a] > period - 2.05 * self.h
                add = torch.zeros(self.d, 1, device=DEV, dtype=torch.float64)
                add[a] = period
                xj, src = (torch.cat([xj, xj[:, lo] + add, xj[:, hi] - add], 1),
                           torch.cat([src, src[lo], src[hi]]))
        i, j, dx, r = pairs(self.x, xj, 2 * self.h, True)
        self.i, self.j, self.r = i, (j if src is None else src[j]), r
        self.e = [q / r for q in dx]
        self.W, self.dWV = kernel.W(r), kernel.dW(r) * self.vol
        self.wi = None
        if self.wall is not None:
            # only the wall near the fluid can have pairs
            self.wi, self.wj, dx, self.wr = pairs(self.x, self.wall, 2 * self.h, False)
            self.we = [q / self.wr for q in dx]
            self.wW, self.wdWV = kernel.W(self.wr), kernel.dW(self.wr) * self.vol
            self.wn = [self.nw[a][self.wj] for a in range(self.d)]

    def advection_dt(self, U_ref, prior):
        a = (self.F + prior).square().sum(0).sqrt() * 4.0 * self.h / self.m
        m = float(torch.maximum(self.v.square().sum(0), a).max())
        return 0.25 * self.h / max(math.sqrt(m), U_ref)

    def acoustic_dt(self):
        return 0.6 * self.h / (self.c0 + math.sqrt(float(self.v.square().sum(0).max())))

    def density(self, kernel, free_surface):
        s0 = lattice_sum(self.d, kernel, self.dp)
        rs = (onto(self.n, self.i, self.W) + kernel.fW) / s0
        if self.wi is not None:
            rs = rs + onto(self.n, self.wi, self.wW) / s0
        self.rho = torch.clamp(rs, min=1.0) if free_surface else rs

    def gravity_force(self):
        return self.m * torch.tensor(self.g[:self.d], device=DEV, dtype=torch.float64)[:, None]

    def first(self, dt, prior):
        i, j, Z = self.i, self.j, self.c0
        self.rho = self.rho + self.rate * (0.5 * dt)
        self.p = p = self.c0 ** 2 * (self.rho - 1.0)
        rate = onto(self.n, i, (p[i] - p[j]) / Z * self.dWV) * self.rho
        s = (p[i] + p[j]) * self.dWV
        F = torch.stack([-onto(self.n, i, s * e) for e in self.e])
        if self.wi is not None:
            wi = self.wi
            face = sum((prior[a].expand(self.n)[wi] / self.m) * -self.we[a] for a in range(self.d))
            pw = p[wi] + self.rho[wi] * self.wr * torch.clamp(face, min=0.0)
            s = (p[wi] + pw) * self.wdWV
            F = F - torch.stack([onto(self.n, wi, s * e) for e in self.we])
            rate = rate + onto(self.n, wi, (p[wi] - pw) / Z * self.wdWV) * self.rho
        self.rate = rate
        self.F = self.F + F * self.vol
        self.x = self.x + self.v * (0.5 * dt)
        self.v = self.v + (prior + self.F) / self.m * dt

    def second(self, dt, riemann=True):
        i, j, Z = self.i, self.j, self.c0
        u = sum((self.v[a][i] - self.v[a][j]) * self.e[a] for a in range(self.d))
        rate = onto(self.n, i, u * self.dWV)
        F = torch.zeros_like(self.F)
        if riemann:
            s = jump(Z, self.c0, u) * self.dWV
            F = torch.stack([onto(self.n, i, s * e) for e in self.e])
        if self.wi is not None:
            wi = self.wi
            ve = sum(self.v[a][wi] * self.we[a] for a in range(self.d))
            vn = sum(self.v[a][wi] * self.wn[a] for a in range(self.d))
            sgn = torch.sign(sum(self.we[a] * self.wn[a] for a in range(self.d)))
            rate = rate + onto(self.n, wi, 2.0 * ve * self.wdWV)
            s = jump(Z, self.c0, 2.0 * sgn * vn) * self.wdWV * sgn
            F = F + torch.stack([onto(self.n, wi, s * q) for q in self.wn])
        self.rate = self.rate + rate * self.rho
        self.F = F * self.vol
        self.rho = self.rho + self.rate * (0.5 * dt)
        self.x = self.x + self.v * (0.5 * dt)

    def dam_break_step(self, U_ref, style=0):
        k = Kernel(self.d, self.h)
        self.configure(k)
        prior = self.gravity_force()
        Dt = self.advection_dt(U_ref, prior)
        self.density(k, True)
        t, dt = 0.0, 0.0
        while t < Dt:
            if style == 0:
                dt = self.acoustic_dt()
            self.first(dt, prior)
            self.second(dt)
            if style == 1:
                dt = self.acoustic_dt()
            t += dt
        return Dt

    def vortex_step(self, t):
        k = Kernel(self.d, self.h)
        self.configure(k, t.L)
        Dt = self.advection_dt(max(t.U, t.mu / self.h), torch.zeros_like(self.F))
        self.density(k, False)
        i, j = self.i, self.j
        c = 2.0 * t.mu * self.dWV / (self.r + 0.01 * self.h)
        prior = torch.stack([onto(self.n, i, c * (self.v[a][i] - self.v[a][j])) for a in range(self.d)]) * self.vol
        inc = torch.stack([-2.0 * onto(self.n, i, self.dWV * e) for e in self.e])
        lim = torch.clamp(100.0 * self.h ** 2 * inc.square().sum(0), max=1.0)
        self.x = self.x + 0.2 * self.h ** 2 * lim * inc
        s = 0.0
        while s < Dt:
            dt = min(self.acoustic_dt(), Dt)
            self.first(dt, prior)
            self.second(dt, riemann=False)
            s += dt
        return Dt

    def ck_step(self, U_ref, rate):
        """The nested CK loop: compression density, correction matrices, averaged Riemann states."""
        d, n, k = self.d, self.n, Kernel(self.d, self.h, tabulated=True)
        self.configure(k)
        i, j, wi = self.i, self.j, self.wi
        comp = kernel_at_zero(k) * self.vol + onto(n, i, self.W) * self.vol + onto(n, wi, self.wW) * self.vol
        comp = torch.clamp(comp, min=1.0)
        V = self.m / comp  # rho = compression
        prior = self.gravity_force()
        Dt = 0.25 * self.h / max(math.sqrt(float(self.v.square().sum(0).max())), U_ref)
        dWV = self.dWV / self.vol * V[j]
        # free-surface indication; every particle counts as a previous surface particle
        thr = {2: 0.75 * 2, 3: 0.75 * 3}[d]
        pd = -onto(n, i, dWV * self.r)
        pd = pd - onto(n, wi, self.wdWV * self.wr)
        near = onto(n, i, ((pd[j] < thr) & (self.r < self.h)).double()) > 0
        surface = torch.where((pd > thr) & ~near, 0, 1).to(torch.int32)
        B = torch.zeros(n, d, d, device=DEV, dtype=torch.float64)
        for a in range(d):
            for b in range(d):
                B[:, a, b] = -(onto(n, i, self.r * self.e[a] * dWV * self.e[b])
                               + onto(n, wi, self.wr * self.we[a] * self.wdWV * self.we[b]))
        det = torch.linalg.det(B)
        wgt = det / (det + torch.clamp(0.5 - det, min=0.0))
        eye = torch.eye(d, device=DEV, dtype=torch.float64)
        inv = torch.linalg.inv(B.transpose(1, 2) @ B + 1e-8 * eye) @ B.transpose(1, 2)
        B = wgt[:, None, None] * inv + (1.0 - wgt)[:, None, None] * eye
        dpos, Z = torch.zeros_like(self.x), self.c0

        def apply(at, e):
            M = B[at]
            return [sum(M[:, a, b] * e[b] for b in range(d)) for a in range(d)]

        bi, bj, bw = apply(i, self.e), apply(j, self.e), apply(wi, self.we)
        s = 0.0
        while s < Dt:
            tot = (self.F + prior).square().sum(0).sqrt()
            fast = torch.maximum(self.c0 + self.v.square().sum(0).sqrt(), (4.0 * self.h * tot / self.m).sqrt())
            dt = 0.6 * self.h / float(fast.max())
            comp = comp + 0.5 * dt * rate
            p = self.c0 ** 2 * (comp - 1.0)
            dpos = dpos + self.v * (0.5 * dt)
            F = torch.stack([-onto(n, i, (p[i] * bj[a] + p[j] * bi[a]) * dWV) for a in range(d)])
            rate = onto(n, i, (p[i] - p[j]) / Z * dWV) * comp
            face = sum(-prior[a].expand(n)[wi] / self.m * self.we[a] for a in range(d))
            pw = p[wi] + comp[wi] * self.wr * torch.clamp(face, min=0.0)
            F = F - torch.stack([onto(n, wi, (p[wi] + pw) * bw[a] * self.wdWV) for a in range(d)])
            rate = rate + onto(n, wi, (p[wi] - pw) / Z * self.wdWV) * comp
            self.F = self.F + F * V
            self.v = self.v + (prior + self.F) / self.m * dt
            v = self.v
            dpos = dpos + v * (0.5 * dt)
            dv = [v[a][i] - v[a][j] for a in range(d)]
            div = onto(n, i, sum(dv[a] * bi[a] for a in range(d)) * dWV)
            pj = jump(Z, self.c0, sum(dv[a] * self.e[a] for a in range(d))) * dWV
            F = torch.stack([onto(n, i, pj * self.e[a]) for a in range(d)])
            div = div + onto(n, wi, sum(2.0 * v[a][wi] * bw[a] for a in range(d)) * self.wdWV)
            sgn = torch.sign(sum(self.we[a] * self.wn[a] for a in range(d)))
            pj = jump(Z, self.c0, sum(2.0 * v[a][wi] * sgn * self.wn[a] for a in range(d))) * self.wdWV
            F = F + torch.stack([onto(n, wi, pj * sgn * self.wn[a]) for a in range(d)])
            self.F = F * V
            rate = rate + div * comp
            comp = comp + 0.5 * dt * rate
            s += dt
        return {"position": self.x + dpos, "velocity": self.v, "density": comp, "pressure": p, "force": self.F,
                "rate": rate, "correction": B.permute(1, 2, 0).reshape(d * d, n), "indicator": surface, "steps": Dt}


def kernel_at_zero(k):
    return float(k.W(torch.zeros(1, device=DEV, dtype=torch.float64)))


def exact(case, seed):
    kind, d = case["kind"], case["dim"]
    if kind == "batch":
        out = {}
        for q, t in enumerate(instances(case, seed)):
            x = torch.from_numpy(np.ascontiguousarray(lattice(t, "water").T)).to(DEV)
            zero = torch.zeros_like(x)
            f = Flow(d, t.dp, t.c0, t.gravity, {"Position": x, "Velocity": zero, "Force": zero,
                                                "Density": zero[0] + 1.0, "DensityChangeRate": zero[0]}, t)
            for _ in range(case["steps"]):
                f.dam_break_step(t.U_ref)
            out["%02d" % q] = [f.x.t(), f.v.t(), f.rho, f.p]
        return out
    if kind in ("tg-mixed", "tg-fp64"):
        t = vortex_case(case)
        f = Flow(d, t.dp, t.c0, (0.0,) * 3, vortex(t, seed))
        Dt = f.vortex_step(t)
        if kind == "tg-mixed":
            x = torch.where(f.x < 0, f.x + t.L, f.x)
            x = torch.where(x > t.L, x - t.L, x)
            return {"position": x, "velocity": f.v, "density": f.rho, "pressure": f.p}
        return {"position": f.x, "velocity": f.v, "density": f.rho, "pressure": f.p, "force": f.F, "rate": f.rate,
                "steps": Dt}
    t = tank(case)
    st = flow(t, seed)
    f = Flow(d, t.dp, t.c0, t.gravity, st, t)
    if kind == "ck":
        return f.ck_step(t.U_ref, 0.05 * torch.sin(37.0 * st["Position"][0]))
    Dt = f.dam_break_step(t.U_ref, t.loop_style)
    if kind == "rows":
        return {"position": f.x.t(), "velocity": f.v.t(), "density": f.rho, "pressure": f.p}
    if kind == "mixed":
        return {"position": f.x, "velocity": f.v, "density": f.rho, "pressure": f.p}
    out = {"position": f.x, "velocity": f.v, "density": f.rho, "pressure": f.p, "force": f.F, "rate": f.rate,
           "steps": Dt}
    if kind == "probes":
        k = Kernel(d, f.h)
        o = torch.tensor(t.observers, device=DEV, dtype=torch.float64).t().contiguous()
        i, j, _, r = pairs(o, st["Position"], 2 * f.h, False)
        w = k.W(r)
        out["probes"] = onto(o.shape[1], i, w * f.p[j]) / onto(o.shape[1], i, w)
        out["energy"] = float((0.5 * f.m * f.v.square().sum(0)).sum()
                              - sum(f.m * t.gravity[a] * f.x[a].sum() for a in range(d)))
    return out
