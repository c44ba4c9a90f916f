"""The work a program has this framework do, as cases that can be timed and
compared: simulation steps over the range of grids, boundaries, storage types
and solvers, batches, the warm-start network's prediction and gradients, and
the headless viewer's frame.

`listed()` names the cases, `draw(rng)` makes more of the same ranges,
`prepare` builds what a program holds before the call, `run` makes one pass
through the public entry points, `work` counts what the pass cannot do
without, and `exact` computes the same outputs in 64 bits with plain torch.

Every simulation case is a running plume: two seeded Gaussian sources near the
floor with an upward force, a smooth flow of about one cell per step and the
uniform velocity perturbation of the 64^3 scene, advanced by one step before
the first pass. A solve that runs until a tolerance has a budget of
sweeps as well, which a developing plume uses up: the passes then cost the same
however far the plume has come.
"""

from __future__ import annotations

import importlib
import math
import pathlib

import numpy as np
import torch

sf = importlib.import_module("stable-fluids_b200")

DT, VISCOSITY, DIFFUSION = 0.1, 1e-4, 1e-5  # the coefficients of every scene of this repository
WEIGHTS = pathlib.Path(__file__).resolve().parent.parent / "stable-fluids_b200" / "weights" / "warmstart_128.npy"
BATCH_SIZES = (32, 48, 64, 96, 128)


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ------------------------------------------------------------------ the cases --
def _step(name, n, diffuse, pressure, walls="stam", scheme="rbgs", storage="fp32", solve="fixed", budget=0):
    return {"name": name, "kind": "step", "nx": n[0], "ny": n[1], "nz": n[2], "diffuse": diffuse, "pressure": pressure, "walls": walls, "scheme": scheme, "storage": storage, "solve": solve, "budget": budget}


def listed():
    return [
        # the smallest grid of the batched workload, stepped alone: interactive use, latency and launches
        _step("step_32", (32, 32, 32), 20, 40),
        # the plain method's small configuration (64^3, 20 / 40 iterations, Stam walls)
        _step("step_64", (64, 64, 64), 20, 40),
        # odd sides: no row is a whole number of vectors (the tiled odd grid of the parity tests)
        _step("step_odd_181x47x29", (181, 47, 29), 20, 40),
        # the reference benchmark's default grid, iterations and boundaries
        _step("step_128x160x128", (128, 160, 128), 24, 96, walls="benchmark"),
        # the plain method at GPU scale (256^3, 20 / 80 iterations)
        _step("step_256", (256, 256, 256), 20, 80),
        # the mixed-precision configuration: BF16 storage at 384^3
        _step("step_bf16_384", (384, 384, 384), 20, 80, storage="bf16"),
        # Jacobi from the previous pressure until the relative residual is 1e-3, within a budget of sweeps
        _step("step_jacobi_tol_128", (128, 128, 128), 20, 80, scheme="jacobi", solve="previous", budget=512),
        # the headline: Jacobi from the learned warm start until 1e-3, at 256^3
        _step("step_learned_256", (256, 256, 256), 20, 80, scheme="jacobi", solve="learned", budget=512),
        # several independent simulations of uneven sizes in one batch step (the default layout)
        {"name": "batch_12", "kind": "batch", "count": 12, "diffuse": 20, "pressure": 40},
        # the network asked for a start directly, on a grid that fills no tile exactly
        {"name": "predict_148x100x60", "kind": "predict", "nx": 148, "ny": 100, "nz": 60},
        # one training pair: loss and every parameter's gradient, at the training resolution
        {"name": "gradients_128", "kind": "gradients", "nx": 128, "ny": 128, "nz": 128},
        # one frame of the headless viewer: the scene's forces, a step, the volume rendered
        {"name": "frame_96x128x96", "kind": "frame", "nx": 96, "ny": 128, "nz": 96, "diffuse": 20, "pressure": 40, "width": 1280, "height": 720, "march": 192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("step", "jacobi", "tolerance", "batch", "predict", "gradients", "frame"), (9, 2, 2, 2, 2, 1, 2))[0]
    if kind in ("step", "jacobi", "tolerance"):
        while True:
            n = [_log_int(rng, 12, 320 if kind == "step" else 200) for _ in range(3)]
            multiple = rng.choice((1, 4, 8, 8))
            n[0] = max(multiple, n[0] // multiple * multiple)
            walls = rng.choice(("stam", "benchmark", "mixed"))
            # an odd periodic side has no red-black colouring: its results depend on the order of the threads
            n[0] += n[0] % 2 if walls == "benchmark" else 0
            n[2] += n[2] % 2 if walls != "stam" else 0
            if n[0] * n[1] * n[2] <= 256 ** 3:
                break
        c = _step("", n, rng.randint(10, 24), rng.randint(20, 96), walls=walls)
        del c["name"]
        if kind == "step" and rng.random() < 0.25:
            c["storage"] = "bf16"
        if kind != "step":
            c["scheme"] = "jacobi"
        if kind == "tolerance":
            c["solve"], c["budget"] = "previous", 16 * rng.randint(4, 40)
        return c
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(3, 12), "diffuse": rng.randint(10, 24), "pressure": rng.randint(20, 60)}
    if kind == "frame":
        return {"kind": "frame", "nx": 8 * rng.randint(4, 16), "ny": rng.randint(32, 160), "nz": 2 * rng.randint(16, 64), "diffuse": rng.randint(10, 24), "pressure": rng.randint(20, 96), "width": rng.randint(320, 1920), "height": rng.randint(240, 1080), "march": rng.randint(64, 256)}
    n = [4 * max(2, _log_int(rng, 16, 160 if kind == "predict" else 128) // 4) for _ in range(3)]
    return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2]}


# ------------------------------------------------------------------ the inputs --
def _f32(v):
    return float(np.float32(v))


def _walls(kind):
    if kind == "stam":
        return sf.scenes.stam_walls()
    if kind == "benchmark":
        return sf.scenes.benchmark_walls()
    # a moving floor, an outflow with a prescribed pressure, fixed scalar faces, one periodic axis
    flow = sf.scenes.flow_boundary([sf.FLOW_NO_SLIP_WALL, sf.FLOW_OUTFLOW, sf.FLOW_NO_SLIP_WALL, sf.FLOW_FREE_SLIP_WALL, sf.FLOW_PERIODIC, sf.FLOW_PERIODIC],
                                   velocities=[(0, 0, 0), (0, 0, 0), (0.02, 0, -0.01), (0, 0, 0), (0, 0, 0), (0, 0, 0)], pressures=[0, 0.001, 0, 0, 0, 0])
    scalar = sf.scenes.scalar_boundary([sf.SCALAR_FIXED_VALUE, sf.SCALAR_ZERO_FLUX, sf.SCALAR_FIXED_VALUE, sf.SCALAR_ZERO_FLUX, sf.SCALAR_PERIODIC, sf.SCALAR_PERIODIC], values=[0.25, 0, 0.5, 0, 0, 0])
    return flow, scalar


def _generator(seed):
    return torch.Generator(device=_dev()).manual_seed(seed)


def _smooth(g, shape, modes=4):
    """A sum of random low-frequency cosines, about unit amplitude."""
    nz, ny, nx = shape
    r = torch.rand((modes, 6), generator=g, device=_dev())
    ax = [(torch.arange(m, device=_dev(), dtype=torch.float32) + 0.5) / m for m in (nz, ny, nx)]
    out = torch.zeros(shape, device=_dev())
    for k in range(modes):
        f = [torch.cos(math.pi * (torch.floor(1 + 4 * r[k, a]) * ax[a] + 2 * r[k, 3 + a])) for a in range(3)]
        out += f[0][:, None, None] * f[1][None, :, None] * f[2][None, None, :]
    return out / math.sqrt(modes)


def _plume(n, seed):
    """(density source, force, impulse added to the force of the first step)"""
    nx, ny, nz = n
    g = _generator(seed)
    shape = (nz, ny, nx)
    radius = min(8.0, max(1.5, min(n) / 16.0))
    z, y, x = (torch.arange(m, device=_dev(), dtype=torch.float32) + 0.5 for m in (nz, ny, nx))
    source, up = torch.zeros(shape, device=_dev()), torch.zeros(shape, device=_dev())
    for _ in range(2):
        r = torch.rand(3, generator=g, device=_dev())
        cx, cz = radius + 1 + r[0] * (nx - 2 * radius - 2), radius + 1 + r[1] * (nz - 2 * radius - 2)
        r2 = (x - cx)[None, None, :] ** 2 + (y - (radius + 2))[None, :, None] ** 2 + (z - cz)[:, None, None] ** 2
        blob = torch.where(r2 <= radius * radius, torch.exp(-2.0 * r2 / (radius * radius)), torch.zeros((), device=_dev()))
        source += 10.0 * blob
        up += (1.0 + 9.0 * r[2]) * blob
    h = 1.0 / nx
    force = (torch.zeros(shape, device=_dev()), up, torch.zeros(shape, device=_dev()))
    impulse = [(h / DT * _smooth(g, shape) + 0.02 * (torch.rand(shape, generator=g, device=_dev()) - 0.5)) / DT for _ in range(3)]
    return source, force, impulse


def _options(case):
    o = sf.default_options()
    if case.get("scheme") == "jacobi":
        o.scheme = sf.SCHEME_JACOBI
    if case.get("storage") == "bf16":
        o.storage = sf.STORAGE_BF16
    solve = case.get("solve", "fixed")
    if solve != "fixed":
        o.warm_start = sf.WARM_START_LEARNED if solve == "learned" else sf.WARM_START_PREVIOUS
        o.residual_tolerance = 1e-3
        o.max_pressure_iterations = case["budget"]
        o.residual_check_interval = 16
        o.warm_start_trial_iterations = 16
    return o


def _simulation(case, walls="stam"):
    flow, scalar = _walls(walls)
    n = (case["nx"], case["ny"], case["nz"])
    config = sf.scenes.make_config(n, _f32(1.0 / n[0]), DT, VISCOSITY, case["diffuse"], case["pressure"], flow)
    return sf.Simulation(config, [sf.ScalarFieldDesc(diffusion=DIFFUSION, dissipation=0.0, initial_value=0.0, boundary=scalar)], [sf.VectorFieldDesc(usage=sf.VECTOR_FIELD_FORCE)], options=_options(case))


def _start(sim, case, seed, step):
    """The plume's inputs and its first step (the one with the impulse)."""
    source, force, impulse = _plume((case["nx"], case["ny"], case["nz"]), seed)
    first = [f + i for f, i in zip(force, impulse)]
    torch.cuda.synchronize()
    sim.set_scalar_source(sim.scalar_handles[0], source)
    sim.set_vector(sim.vector_handles[0], *first)
    if step:
        sim.step()
        sim.set_vector(sim.vector_handles[0], *force)
    sim.synchronize()
    return force


def _batch_cases(case, seed):
    # every size of the range, the larger ones rarer: the same sizes for every seed
    sizes = [BATCH_SIZES[(k * 3) % 5] if k % 4 else 64 for k in range(case["count"])]
    return [({"nx": s, "ny": s, "nz": s, "diffuse": case["diffuse"], "pressure": case["pressure"]}, 1000 * seed + k) for k, s in enumerate(sizes)]


def _network():
    net = sf.WarmStartNetwork(seed=0)
    net.set_parameters(np.load(WEIGHTS))
    return net


def _pair(case, seed):
    """(divergence, previous pressure, converged pressure): smooth pressures and a divergence with fine detail."""
    shape = (case["nz"], case["ny"], case["nx"])
    g = _generator(seed)
    b = 0.2 * _smooth(g, shape, 8) + 0.05 * torch.randn(shape, generator=g, device=_dev())
    scale = 1.0 / case["nx"]
    previous = scale * _smooth(g, shape)
    return b, previous, previous + 0.3 * scale * _smooth(g, shape)


def _camera(case):
    ext = np.array([case["nx"], case["ny"], case["nz"]], np.float64) / case["nx"]
    centre = ext / 2
    eye = centre + np.array([0.35, 0.25, -1.6]) * ext.max()
    forward = (centre - eye) / np.linalg.norm(centre - eye)
    right = np.cross([0.0, 1.0, 0.0], forward)
    right /= np.linalg.norm(right)
    up = np.cross(forward, right)
    c = {"eye": eye, "right": right, "up": up, "forward": forward, "volume_min": np.zeros(3), "volume_max": ext, "color_a": np.array([0.1, 0.2, 0.9]), "color_b": np.array([1.0, 0.6, 0.1])}
    c = {k: [_f32(x) for x in v] for k, v in c.items()}
    c.update(aspect=_f32(case["width"] / case["height"]), tan_half_fov=0.5, value_scale=1.0, density=6.0, value_min=0.0, value_max=4.0, ortho_height=1.0, steps=case["march"], projection=0, width=case["width"], height=case["height"])
    return c


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        sim = _simulation(case, case["walls"])
        state = {"kind": kind, "sim": sim}
        if case["solve"] == "learned":
            state["net"] = _network()
            state["net"].attach(sim)
        _start(sim, case, seed, step=True)
        return state
    if kind == "batch":
        sims = []
        forces = []
        for c, s in _batch_cases(case, seed):
            sims.append(_simulation(c))
            forces.append(_start(sims[-1], c, s, step=False))
        batch = sf.Batch(sims)
        batch.step()
        for sim, force in zip(sims, forces):
            sim.set_vector(sim.vector_handles[0], *force)
            sim.synchronize()
        return {"kind": kind, "batch": batch, "sims": sims}
    if kind == "frame":
        sim = _simulation(case, "benchmark")
        sim.plume_scene_setup()
        sim.plume_scene_forces(seed % 997)
        sim.step()
        p = sf.B200VolumeRender()
        for k, v in _camera(case).items():
            if isinstance(v, list):
                getattr(p, k)[:] = v
            else:
                setattr(p, k, v)
        image = torch.empty((case["height"], case["width"], 4), device=_dev())
        torch.cuda.synchronize()
        return {"kind": kind, "sim": sim, "camera": p, "image": image, "frame": seed % 997}
    return {"kind": kind, "net": _network(), "h": _f32(1.0 / case["nx"]), "pair": _pair(case, seed)}


def _views(state, sim):
    """(vx, vy, vz, density): views of the simulation's memory, which each of them keeps alive"""
    views = (*sim.view(sf.VIEW_FLOW_VELOCITY), sim.view(sf.VIEW_SCALAR_FIELD_DATA, sim.scalar_handles[0]))
    for v in views:
        v.owner = state
    return views


def run(state):
    kind = state["kind"]
    if kind == "step":
        sim = state["sim"]
        sim.step()
        vx, vy, vz, density = _views(state, sim)
        pressure = sim.view(sf.VIEW_FLOW_PRESSURE)
        pressure.owner = state
        return {"density": density, "vx": vx, "vy": vy, "vz": vz, "pressure": pressure}
    if kind == "batch":
        state["batch"].step()
        return [_views(state, sim) for sim in state["sims"]]
    if kind == "frame":
        sim = state["sim"]
        state["frame"] += 1
        sim.plume_scene_forces(state["frame"])
        sim.step()
        image = sim.render_volume(sf.VIEW_SCALAR_FIELD_DATA, state["camera"], sim.scalar_handles[0], out=state["image"])
        density = sim.view(sf.VIEW_SCALAR_FIELD_DATA, sim.scalar_handles[0])
        density.owner = state
        return {"image": image, "density": density}
    b, previous, target = state["pair"]
    if kind == "predict":
        return state["net"].predict(b, previous, state["h"])
    loss, gradients = state["net"].gradients(b, previous, target, state["h"])
    return {"loss": loss, "gradients": gradients}


_LAYERS = ((16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16), (16, 16))
_LEVEL = (0, 0, 1, 1, 2, 2, 1, 1, 0, 0, 0)


def work(case):
    if case["kind"] == "batch":
        parts = [work({**c, "kind": "step"}) for c, _ in _batch_cases(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    cells = case["nx"] * case["ny"] * case["nz"]
    net = sum(54 * ci * co / 8 ** lv for (ci, co), lv in zip(_LAYERS, _LEVEL)) * cells
    if case["kind"] == "predict":
        return {"bytes": 12 * cells, "flops": net}
    if case["kind"] == "gradients":
        return {"bytes": 12 * cells, "flops": 3 * net}
    # state, source and forces read, state and the diagnostic fields written; 9 operations a cell and iteration, about 300 for the rest
    advected = 2 if case.get("storage") == "bf16" else 4
    sweeps = 4 * case["diffuse"] + (case["pressure"] if case.get("solve", "fixed") == "fixed" else case["budget"])
    w = {"bytes": (8 * advected + 28) * cells, "flops": (9.0 * sweeps + 300) * cells}
    if case.get("solve") == "learned":
        w["flops"] += net
    if case["kind"] == "frame":
        w["bytes"] += 16 * case["width"] * case["height"]
        w["flops"] += 20.0 * case["width"] * case["height"] * case["march"]
    return w


# ------------------------------------------------------- the same in 64 bits --
def _along(t, axis, sl):
    i = [slice(None)] * 3
    i[2 - axis] = sl
    return t[tuple(i)]


class _Step64:
    """One simulation in FP64 on dense (nz, ny, nx) tensors."""

    def __init__(self, case, walls):
        self.case = case
        self.n = (case["nx"], case["ny"], case["nz"])
        self.shape = self.n[::-1]
        self.h, self.dt = _f32(1.0 / case["nx"]), _f32(DT)
        flow, scalar = _walls(walls)
        names = [f[0] for f in type(flow)._fields_]
        self.flow, self.scalar = [getattr(flow, k) for k in names], [getattr(scalar, k) for k in names]
        self.periodic = [self.flow[2 * a].type == sf.FLOW_PERIODIC for a in range(3)]
        self.s_periodic = [self.scalar[2 * a].type == sf.SCALAR_PERIODIC for a in range(3)]
        zero = lambda: torch.zeros(self.shape, dtype=torch.float64, device=_dev())  # noqa: E731
        self.v, self.p, self.rho = [zero() for _ in range(3)], zero(), zero()
        z, y, x = (torch.arange(m, device=_dev()) for m in self.shape)
        self.red = (x[None, None, :] + y[None, :, None] + z[:, None, None]) % 2 == 0
        self.iterations = []

    # (periodic?, [(mode, constant) per face]) of a field: "copy", "const" or "reflect" about half the constant
    def rule(self, what):
        if what == "p":
            return self.periodic, [("const", f.pressure) if f.type == sf.FLOW_OUTFLOW else ("copy", 0.0) for f in self.flow]
        if what == "s":
            return self.s_periodic, [("const", f.value) if f.type == sf.SCALAR_FIXED_VALUE else ("copy", 0.0) for f in self.scalar]
        out = []
        for k, f in enumerate(self.flow):
            copy = f.type == sf.FLOW_OUTFLOW or (f.type == sf.FLOW_FREE_SLIP_WALL and what != k // 2)
            out.append(("copy", 0.0) if copy else ("reflect", 2.0 * (f.velocity_x, f.velocity_y, f.velocity_z)[what]))
        return self.periodic, out

    def pad(self, t, axis, rule):
        """t with one ghost layer on both sides of one axis."""
        periodic, faces = rule
        lo, hi = _along(t, axis, slice(0, 1)), _along(t, axis, slice(-1, None))
        if periodic[axis]:
            return torch.cat([hi, t, lo], 2 - axis)

        def ghost(face, own):
            mode, k = face
            return own if mode == "copy" else torch.full_like(own, k) if mode == "const" else k - own

        return torch.cat([ghost(faces[2 * axis], lo), t, ghost(faces[2 * axis + 1], hi)], 2 - axis)

    def neighbours(self, t, rule):
        out = None
        for axis in range(3):
            q = self.pad(t, axis, rule)
            s = _along(q, axis, slice(0, -2)) + _along(q, axis, slice(2, None))
            out = s if out is None else out.add_(s)
        return out

    def gradient(self, t, axis, rule):
        q = self.pad(t, axis, rule)
        return (_along(q, axis, slice(2, None)) - _along(q, axis, slice(0, -2))) * (0.5 / self.h)

    def solve(self, x, update, rule, count, jacobi):
        for _ in range(count):
            if jacobi:
                x = update(self.neighbours(x, rule))
            else:
                for red in (True, False):
                    x = torch.where(self.red == red, update(self.neighbours(x, rule)), x)
        return x

    # ---- semi-Lagrangian gathers, a slab of planes at a time
    def corners(self, pos, periodic):
        g = []
        for a in range(3):
            q = torch.remainder(pos[a], self.n[a] * self.h) if periodic[a] else pos[a]
            g.append(q / self.h - 0.5)
        base = [torch.floor(q) for q in g]
        t = [q - b for q, b in zip(g, base)]
        return [b.clamp(-2, m).long() for b, m in zip(base, self.n)], t

    def lerp8(self, values, t):
        for a in range(3):
            values = [u + (w - u) * t[a] for u, w in zip(values[0::2], values[1::2])]
        return values[0]

    def index(self, c):
        return c[0] + self.n[0] * (c[1] + self.n[1] * c[2])

    def sample_velocity(self, pos, components):
        base, t = self.corners(pos, self.periodic)
        rules = [self.rule(k)[1] for k in range(3)]
        got = [[] for _ in components]
        for k in range(8):
            c = [base[a] + ((k >> a) & 1) for a in range(3)]
            face = torch.full_like(c[0], -1)
            for a in range(3):
                if self.periodic[a]:
                    c[a] = torch.where(face < 0, torch.remainder(c[a], self.n[a]), c[a])
                else:
                    face = torch.where((face < 0) & (c[a] < 0), 2 * a, torch.where((face < 0) & (c[a] >= self.n[a]), 2 * a + 1, face))
            i = self.index([c[a].clamp(0, self.n[a] - 1) for a in range(3)])
            for j, comp in enumerate(components):
                f = self.v[comp].reshape(-1)[i]
                for q, (mode, const) in enumerate(rules[comp]):
                    if mode == "reflect":
                        f = torch.where(face == q, const - f, f)
                got[j].append(f)
        return [self.lerp8(v, t) for v in got]

    def sample_scalar(self, q, pos):
        base, t = self.corners(pos, self.s_periodic)
        got = []
        for k in range(8):
            c = [base[a] + ((k >> a) & 1) for a in range(3)]
            fixed = torch.full_like(t[0], math.nan)
            for a in range(3):
                if self.s_periodic[a]:
                    c[a] = torch.remainder(c[a], self.n[a])
                    continue
                for side, out in ((0, c[a] < 0), (1, c[a] >= self.n[a])):
                    f = self.scalar[2 * a + side]
                    if f.type == sf.SCALAR_FIXED_VALUE:
                        fixed = torch.where(out & fixed.isnan(), torch.full_like(fixed, f.value), fixed)
                c[a] = c[a].clamp(0, self.n[a] - 1)
            v = q.reshape(-1)[self.index(c)]
            got.append(torch.where(fixed.isnan(), v, fixed))
        return self.lerp8(got, t)

    def advect(self, sample):
        """`sample(back-traced positions)` for every cell, midpoint traces in self.v."""
        nx, ny, nz = self.n
        planes = max(1, (4 << 20) // (nx * ny))
        x, y, z = (((torch.arange(m, device=_dev(), dtype=torch.float64) + 0.5) * self.h) for m in self.n)
        parts = []
        for z0 in range(0, nz, planes):
            shape = (min(planes, nz - z0), ny, nx)
            at = [x[None, None, :].expand(shape), y[None, :, None].expand(shape), z[z0:z0 + planes, None, None].expand(shape)]
            v0 = [v[z0:z0 + planes] for v in self.v]
            v1 = self.sample_velocity([p - 0.5 * self.dt * v for p, v in zip(at, v0)], (0, 1, 2))
            parts.append(sample([p - self.dt * v for p, v in zip(at, v1)]))
        return [torch.cat([p[k] for p in parts]) for k in range(len(parts[0]))]

    def residual(self, p, b):
        r = b - (self.neighbours(p, self.rule("p")) - 6.0 * p)
        if not any(f.type == sf.FLOW_OUTFLOW for f in self.flow):
            r, b = r - b.mean(), b - b.mean()
        return float(r.norm() / b.norm()) if float(b.norm()) > 0 else 0.0

    def step(self, source, force, predict=None):
        c, dt, h = self.case, self.dt, self.h
        jacobi = c.get("scheme") == "jacobi"
        self.v = [v + dt * f.double() for v, f in zip(self.v, force)]
        advected = self.advect(lambda pos: self.sample_velocity(pos, (0, 1, 2)))
        a = dt * _f32(VISCOSITY) / (h * h)
        for k in range(3):
            b = advected[k]
            self.v[k] = self.solve(b, lambda nb, b=b: (b + a * nb) / (1 + 6 * a), self.rule(k), c["diffuse"], jacobi)
        div = sum(self.gradient(self.v[k], k, self.rule(k)) for k in range(3))
        b, rule = h * h * div, self.rule("p")
        update = lambda nb: (nb - b) / 6.0  # noqa: E731
        if c.get("solve", "fixed") == "fixed":
            self.p = self.solve(torch.zeros_like(self.p), update, rule, c["pressure"], jacobi)
        else:
            p, done = self.p, 0
            if predict is not None:  # the better of the two starts after 16 sweeps each
                p, done = self.solve(predict(div, p), update, rule, 16, True), 16
                plain = self.solve(self.p, update, rule, 16, True)
                if self.residual(p, b) > self.residual(plain, b):
                    p = plain
            rel = self.residual(p, b)
            while rel > _f32(1e-3) and done < c["budget"]:
                p = self.solve(p, update, rule, 15, True)
                rel = self.residual(p, b)
                p = self.solve(p, update, rule, 1, True)
                done += 16
            self.p = p
            self.iterations.append(done)
        for k in range(3):
            self.v[k] = self.v[k] - self.gradient(self.p, k, rule)
        q = self.rho + dt * source.double()
        b2 = self.advect(lambda pos: [self.sample_scalar(q, pos)])[0]
        a2 = dt * _f32(DIFFUSION) / (h * h)
        self.rho = self.solve(b2, lambda nb: (b2 + a2 * nb) / (1 + 6 * a2), self.rule("s"), c["diffuse"], jacobi)


def _plume64(case, seed, walls, predict=None):
    s = _Step64(case, walls)
    source, force, impulse = _plume(s.n, seed)
    s.step(source, [f + i for f, i in zip(force, impulse)], predict)
    del impulse
    s.step(source, force, predict)
    return s


# ---- the network: channels-last FP64 activations, patches gathered a few planes at a time
def _patches(x, z0, z1):
    nz, ny, nx, c = x.shape
    slab = torch.zeros((z1 - z0 + 2, ny + 2, nx + 2, c), dtype=x.dtype, device=x.device)
    lo, hi = max(z0 - 1, 0), min(z1 + 1, nz)
    slab[lo - z0 + 1:hi - z0 + 1, 1:-1, 1:-1] = x[lo:hi]
    return torch.cat([slab[d:d + z1 - z0, e:e + ny, f:f + nx] for d in range(3) for e in range(3) for f in range(3)], -1).reshape(-1, 27 * c)


def _slabs(x):
    per = max(1, (1 << 28) // (x.shape[1] * x.shape[2] * x.shape[3] * 27))
    return [(z, min(z + per, x.shape[0])) for z in range(0, x.shape[0], per)]


def _conv(x, w, bias=None):
    """w: (27, cout, cin)"""
    m = w.permute(0, 2, 1).reshape(-1, w.shape[1])
    y = torch.cat([_patches(x, *s) @ m for s in _slabs(x)]).reshape(*x.shape[:3], w.shape[1])
    return y if bias is None else y + bias


def _weight_gradient(x, g):
    dw = sum(_patches(x, *s).T @ g[s[0]:s[1]].reshape(-1, g.shape[3]) for s in _slabs(x))
    return torch.cat([dw.reshape(27, x.shape[3], g.shape[3]).permute(0, 2, 1).reshape(-1), g.sum((0, 1, 2))])


def _pool(x):
    z, y, w, c = x.shape
    return x.reshape(z // 2, 2, y // 2, 2, w // 2, 2, c).sum((1, 3, 5))


def _up(x):
    return x.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)


class _Net64:
    def __init__(self):
        flat, at = torch.from_numpy(np.load(WEIGHTS)).double().to(_dev()), 0
        self.w, self.b = [], []
        for ci, co in _LAYERS:
            self.w.append(flat[at:at + 27 * ci * co].reshape(27, co, ci))
            at += 27 * ci * co
            self.b.append(flat[at:at + co])
            at += co

    def forward(self, div, previous, h):
        b = div.double() * (h * h)
        self.scale = float(1.0 / b.square().mean().sqrt())
        x = torch.zeros((*b.shape, 16), dtype=torch.float64, device=_dev())
        x[..., 0], x[..., 1] = b * self.scale, previous.double() * self.scale
        self.x, self.y = [], []  # every layer's input and output

        def layer(k, t):
            t = _conv(t, self.w[k], self.b[k])
            return t if k == 10 else t.clamp_(min=0.0)

        def chain(k, t):
            for i in (k, k + 1):
                self.x.append(t)
                t = layer(i, t)
                self.y.append(t)
            return t

        e0 = chain(0, x)
        e1 = chain(2, _pool(e0) / 8)
        t = chain(4, _pool(e1) / 8)
        t = chain(6, torch.cat([_up(t), e1], -1))
        t = chain(8, torch.cat([_up(t), e0], -1))
        self.x.append(t)
        return layer(10, t)[..., 0]

    def predict(self, div, previous, h):
        out = previous.double() + self.forward(div, previous, h) / self.scale
        self.x = self.y = None
        return out

    def gradients(self, div, previous, target, h):
        e = self.forward(div, previous, h) - (target.double() - previous.double()) * self.scale
        g = torch.zeros((*e.shape, 16), dtype=torch.float64, device=_dev())
        g[..., 0] = 2.0 / e.numel() * e
        got = [None] * 11

        def back(k, g):
            """The gradient of layer k's input from that of its output."""
            if k < 10:
                g = torch.where(self.y[k] > 0, g, torch.zeros((), dtype=g.dtype, device=g.device))
            got[k] = _weight_gradient(self.x[k], g)
            return _conv(g, self.w[k].flip(0).permute(0, 2, 1)) if k else None

        g = back(8, back(9, back(10, g)))
        skip0 = g[..., 32:]
        g = back(6, back(7, _pool(g[..., :32])))
        skip1 = g[..., 64:]
        g = back(4, back(5, _pool(g[..., :64])))
        g = back(2, back(3, skip1 + _up(g) / 8))
        back(0, back(1, skip0 + _up(g) / 8))
        return float(e.square().mean()), torch.cat(got)


# ---- the viewer's scene and its volume
def _scene_forces(case, frame):
    h = _f32(1.0 / case["nx"])
    ext = [case[k] * h for k in ("nx", "ny", "nz")]
    r = 6.0 * h
    sx, sy, sz = 0.5 * ext[0], 0.13 * ext[1], 0.5 * ext[2]
    x, y, z = ((torch.arange(case[k], device=_dev(), dtype=torch.float64) + 0.5) * h for k in ("nx", "ny", "nz"))
    x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]

    def weight(cy, radius):
        return (1.0 - ((x - sx) ** 2 + (y - cy) ** 2 + (z - sz) ** 2) / (radius * radius)).clamp(min=0.0)

    phase = frame * 0.045
    source = weight(sy, r)
    swirl = 1.65 * math.cos(0.53 * phase) * weight(sy + 0.9 * r, 1.65 * r)
    drift = weight(sy + 1.35 * r, 2.1 * r)
    radial = ((x - sx) ** 2 + (z - sz) ** 2).sqrt()
    inv = torch.where(radial > 1e-5, 1.0 / radial, torch.zeros((), dtype=torch.float64, device=_dev()))
    fx = 1.15 * math.sin(phase) * drift - swirl * (z - sz) * inv
    fz = 0.85 * math.cos(0.71 * phase) * drift + swirl * (x - sx) * inv
    return 32.0 * source, (fx, 7.6 * source, fz)


def _render64(field, c):
    d = _dev()
    v = {k: torch.tensor(c[k], dtype=torch.float64, device=d) for k in ("eye", "right", "up", "forward", "volume_min", "volume_max", "color_a", "color_b")}
    px = (torch.arange(c["width"], device=d, dtype=torch.float64) + 0.5) / c["width"] * 2 - 1
    py = 1 - (torch.arange(c["height"], device=d, dtype=torch.float64) + 0.5) / c["height"] * 2
    ray = v["forward"] + v["right"] * (px * c["aspect"] * c["tan_half_fov"])[None, :, None] + v["up"] * (py * c["tan_half_fov"])[:, None, None]
    ray = ray / ray.norm(dim=-1, keepdim=True)
    inv = 1.0 / torch.where(ray.abs() < 1e-6, torch.where(ray < 0, -1e-6, 1e-6).double(), ray)
    a, b = (v["volume_min"] - v["eye"]) * inv, (v["volume_max"] - v["eye"]) * inv
    t0, t1 = torch.minimum(a, b).amax(-1).clamp(min=0.0), torch.maximum(a, b).amin(-1)
    hit = t1 > t0
    rays, t0 = ray[hit], t0[hit]
    length = (t1[hit] - t0) / c["steps"]
    n = torch.tensor(field.shape[::-1], device=d)
    flat = field.reshape(-1)
    trans, color = torch.ones_like(t0), torch.zeros_like(rays)
    live = torch.ones_like(t0, dtype=torch.bool)
    for i in range(c["steps"]):
        w = v["eye"] + rays * (t0 + (i + 0.5) * length)[:, None]
        q = ((w - v["volume_min"]) / (v["volume_max"] - v["volume_min"])).clamp(0, 1) * (n - 1)
        lo = q.floor()
        t = (q - lo).unbind(-1)
        lo = lo.long()
        hi = torch.minimum(lo + 1, n - 1)
        at = [(lo if not (k >> a) & 1 else hi)[:, a] for k in range(8) for a in range(3)]
        val = [flat[at[3 * k] + n[0] * (at[3 * k + 1] + n[1] * at[3 * k + 2])] for k in range(8)]
        for a in range(3):
            val = [p + (r - p) * t[a] for p, r in zip(val[0::2], val[1::2])]
        level = ((val[0] * c["value_scale"] - c["value_min"]) / (c["value_max"] - c["value_min"])).clamp(0, 1)
        alpha = torch.where(live & (level >= 1e-4), 1.0 - torch.exp(-level * c["density"] * length), torch.zeros_like(level))
        color += (v["color_a"] + level[:, None] * (v["color_b"] - v["color_a"])) * (trans * alpha)[:, None]
        trans = trans * (1.0 - alpha)
        live &= trans >= 0.01
    out = torch.zeros((c["height"], c["width"], 4), dtype=torch.float64, device=d)
    out[hit] = torch.cat([color, (1.0 - trans)[:, None]], -1)
    return out


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        net = _Net64() if case["solve"] == "learned" else None
        s = _plume64(case, seed, case["walls"], predict=None if net is None else lambda div, p: net.predict(div, p, _f32(1.0 / case["nx"])))
        return {"density": s.rho, "vx": s.v[0], "vy": s.v[1], "vz": s.v[2], "pressure": s.p}
    if kind == "batch":
        out = []
        for c, seed_k in _batch_cases(case, seed):
            s = _plume64(c, seed_k, "stam")
            out.append((*s.v, s.rho))
        return out
    if kind == "frame":
        s = _Step64(case, "benchmark")
        for k in range(2):
            source, force = _scene_forces(case, seed % 997 + k)
            s.step(source, force)
        return {"image": _render64(s.rho, _camera(case)), "density": s.rho}
    b, previous, target = _pair(case, seed)
    h = _f32(1.0 / case["nx"])
    if kind == "predict":
        return _Net64().predict(b, previous, h)
    loss, gradients = _Net64().gradients(b, previous, target, h)
    return {"loss": loss, "gradients": gradients}
