"""Timed cases of the SPH engine.

Each case is one call sequence that a host program of the engine makes, on a
scene of the package's own configurations: time steps of every pressure solver
through host buffers (`GpuSystem.step_host`), a restart from a checkpoint, a
sensor plane, a fluid surface, and a batch of scenes through the scene server.

`exact` restates the same update in plain torch with 64-bit numbers (pair
lists instead of kernels); it shares nothing with the engine but the scene.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

for _root in (os.getcwd(), os.path.dirname(os.path.dirname(os.path.abspath(__file__)))):
    _pkg = os.path.join(_root, "fluid-simulation_b200")
    if os.path.isdir(_pkg):
        sys.path.insert(0, _pkg)
        break

from sphgpu import GpuSystem, SceneServer, capi, scenes  # noqa: E402
from sphgpu.fields import build_volume_map_fields  # noqa: E402

QUANTITIES = {"speed": capi.Q_SPEED, "volume": capi.Q_VOLUME, "density": capi.Q_DENSITY}
G = 9.81


# ---- cases -------------------------------------------------------------------
def listed():
    return [
        # the smallest served scene, stepped as the server steps it (step graphs)
        dict(name="iisph_serving_5k", kind="step", scene="serving", solver="IISPH", side=17, precision="f32",
             steps=8, graph=8),
        # a small weakly compressible dam break (8,000 particles, like the repository's first
        # configuration): one 10 ms frame
        dict(name="sesph_dam_8k", kind="step", scene="serving", solver="SESPH", side=20, precision="f32",
             steps=10, graph=0),
        # an ordinary scene with the splitting solver
        dict(name="splitting_dam_30k", kind="step", scene="serving", solver="SESPHwSplitting", side=31,
             precision="f32", steps=5, graph=0),
        # a large served scene, weakly compressible
        dict(name="sesph_serving_195k", kind="step", scene="serving", solver="SESPH", side=58, precision="f32",
             steps=4, graph=0),
        # an ordinary dam break in a volume-map box
        dict(name="iisph_box_133k", kind="step", scene="box", solver="IISPH", side=51, precision="f32", steps=4,
             graph=0),
        # the benchmark scene: the largest single-fluid dam break
        dict(name="iisph_box_1m", kind="step", scene="box", solver="IISPH", side=100, precision="f32", steps=4,
             graph=0),
        # the same kind of scene in 64-bit state (precision studies)
        dict(name="iisph_box_f64_64k", kind="step", scene="box", solver="IISPH", side=40, precision="f64", steps=3,
             graph=0),
        # fluid coupled with eight rigid bodies, CFL steps: restart from a checkpoint, then steps
        dict(name="tank_bodies_282k", kind="step", scene="tank", solver="IISPH", side=79, precision="f32", steps=3,
             graph=0),
        # two fluids in a sphere: restart from a checkpoint, then steps
        dict(name="ball_two_fluids", kind="ball", side=50, precision="f32", steps=3),
        # a sensor plane of a recording
        dict(name="sensor_plane_512", kind="plane", side=60, rows=512, cols=512, quantity="speed"),
        # a triangle-mesh frame of a recording
        dict(name="surface_64k", kind="surface", side=40),
        # a few requests of the scene sweep, served together
        dict(name="server_mix", kind="server", scenes=6, small=5000, large=60000, steps=25),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["serving", "serving", "serving", "box", "box", "tank", "ball", "plane", "surface", "server"])
    if kind == "serving":
        solver = rng.choice(["SESPH", "IISPH", "SESPHwSplitting"])
        side = int(round(_log_uniform(rng, 5e3, 5e5) ** (1.0 / 3.0)))
        steps = rng.randint(1, 10 if side < 40 else 4)
        return dict(kind="step", scene="serving", solver=solver, side=side, precision="f32", steps=steps,
                    graph=rng.choice([0, 0, steps]))
    if kind == "box":
        precision = rng.choice(["f32", "f32", "f64"])
        side = int(round(_log_uniform(rng, 8e3, 8e5 if precision == "f32" else 2e5) ** (1.0 / 3.0)))
        return dict(kind="step", scene="box", solver="IISPH", side=side, precision=precision,
                    steps=rng.randint(1, 4), graph=0)
    if kind == "tank":
        return dict(kind="step", scene="tank", solver="IISPH", side=rng.randint(30, 79), precision="f32",
                    steps=rng.randint(1, 3), graph=0)
    if kind == "ball":
        return dict(kind="ball", side=rng.randint(20, 55), precision=rng.choice(["f32", "f32", "f64"]),
                    steps=rng.randint(1, 3))
    if kind == "plane":
        return dict(kind="plane", side=rng.randint(25, 60), rows=rng.randint(63, 700), cols=rng.randint(63, 700),
                    quantity=rng.choice(list(QUANTITIES)))
    if kind == "surface":
        return dict(kind="surface", side=rng.randint(17, 45))
    return dict(kind="server", scenes=rng.randint(2, 6), small=5000, large=rng.randint(10000, 60000),
                steps=rng.randint(10, 25))


# ---- inputs --------------------------------------------------------------------
def _f32(a):
    return np.asarray(a, np.float32).astype(np.float64)


def _flow(position, seed):
    """A seeded divergence-free sloshing flow, a third as fast as a
    shallow-water wave over the block."""
    rng = np.random.default_rng(seed)
    phase = rng.uniform(0.0, 2.0 * np.pi, 3)
    lo, hi = position.min(axis=0), position.max(axis=0)
    length = float((hi - lo).max())
    speed = 0.3 * math.sqrt(G * length)
    q = 2.0 * np.pi * (position - lo) / length
    v = speed * np.stack([np.sin(q[:, 1] + phase[0]), np.sin(q[:, 2] + phase[1]), np.sin(q[:, 0] + phase[2])], axis=1)
    return _f32(v)


def _serving(solver, side, seed):
    sc = scenes.serving_dam_break(side ** 3, "IISPH" if solver == "IISPH" else "SESPH", seed=seed)
    if solver == "SESPHwSplitting":
        sc.procedures["pressure_solver"] = "SESPHwSplitting"
    return sc


def _scene(case, seed):
    """The case's scene as a flow in progress (see _in_motion)."""
    if case["kind"] == "ball":
        sc = scenes.two_fluid_ball(radius=0.008 * case["side"], spacing=0.008, seed=seed)
    elif case["kind"] in ("plane", "surface") or case["scene"] == "box":
        n = case["side"]
        sc = scenes.dam_break_iisph_box(n_side=n, spacing=0.01, jitter_seed=seed, box=(0.02 * n, 0.01 * n, 0.01 * n))
        sc.cfl_time_step = False
        sc.parameters["time_increment"] = 1e-3
    elif case["scene"] == "tank":
        y = case["side"] * 0.01 + 0.01  # particles across the tank, plus the wall gaps
        sc = scenes.rigid_body_tank(spacing=0.01, tank=(1.5 * y, y, y), fill=0.375 * y, cube_side=0.15 * y,
                                    sphere_radius=0.08 * y, seed=seed)
    else:
        sc = _serving(case["solver"], case["side"], seed)
    return _in_motion(sc, seed)


def _in_motion(sc, seed):
    """The scene as a flow in progress: moving, and with seeded density waves of
    0.5 % over thirty spacings, so that an implicit solver meets a density
    error like the one it works against all along a run (a lattice at rest has
    none, and needs the least sweeps)."""
    wave = 2.0 * np.pi / (30.0 * sc.parameters["rest_density_grid_spacing"])
    phase = np.random.default_rng(seed + 1).uniform(0.0, 2.0 * np.pi, 3)
    sc.position = _f32(sc.position + 0.005 / wave * np.sin(wave * sc.position + phase))
    sc.velocity = _flow(sc.position, seed)
    if sc.procedures["pressure_solver"] in ("IISPH", "IISPHwOST"):
        sc.parameters["max_solver_iterations"] = 100
    return sc


@functools.lru_cache(maxsize=4)
def _fields_of(verts, n_verts, faces, dx, radius):
    v = np.frombuffer(verts, np.float64).reshape(n_verts, 3)
    return build_volume_map_fields(v, np.frombuffer(faces, np.uint32).reshape(-1, 3), dx, radius)


def _fields(sc):
    """(sdf, vm) of a volume-map scene's container: a program builds them once
    per container, whatever fluid it puts in."""
    if sc.procedures["boundary_handling"] != "VolumeMapBoundary":
        return None
    verts, faces = (np.ascontiguousarray(a) for a in sc.mesh)
    return _fields_of(verts.tobytes(), len(verts), faces.tobytes(), 4 * sc.parameters["rest_density_grid_spacing"],
                      sc.parameters["kernel_support_radius"])


def _server_scenes(case, seed):
    n = np.exp(np.linspace(math.log(case["small"]), math.log(case["large"]), case["scenes"]))
    out = []
    for k, target in enumerate(n):
        sc = _serving("SESPH" if k % 2 == 0 else "IISPH", int(round(target ** (1.0 / 3.0))), seed + 1000 * k)
        out.append(_in_motion(sc, seed + k))
    return out


def _plane(case, sc, seed):
    """Points of a vertical sensor plane through the container, as rows x cols
    positions (f32, like the recording's planes)."""
    half = 0.5 * np.asarray(sc.container)
    y = float(np.random.default_rng(seed).uniform(-0.4, 0.4) * half[1])
    z, x = np.meshgrid(np.linspace(-half[2], half[2], case["rows"]), np.linspace(-half[0], half[0], case["cols"]),
                       indexing="ij")
    return np.stack([x, np.full_like(x, y), z], axis=-1).reshape(-1, 3).astype(np.float32)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float64)).pin_memory()


def prepare(case, seed):
    if case["kind"] == "server":
        return {"case": case, "server": SceneServer(), "scenes": _server_scenes(case, seed)}
    sc = _scene(case, seed)
    system: GpuSystem = scenes.build_system(sc, precision=case.get("precision", "f32"), fields=_fields(sc))
    state = {"case": case, "system": system}
    if case["kind"] == "plane":
        state["points"] = _plane(case, sc, seed)
    if case["kind"] == "surface":
        # the renderer's buffers: a lattice cell per 0.375 spacings over the block's faces, and half as many again
        room = int(1.5 * 6 * (case["side"] / 0.375) ** 2) + 1000
        state["vertices"], state["indices"] = np.zeros((room, 6)), np.zeros(6 * room, np.uint32)
    if case["kind"] in ("step", "ball"):
        state["x_out"] = torch.empty(sc.position.shape, dtype=torch.float64).pin_memory()
        state["v_out"] = torch.empty(sc.position.shape, dtype=torch.float64).pin_memory()
        state["x"], state["v"] = (torch.empty(sc.position.shape, dtype=torch.float32) for _ in range(2))
    if case["kind"] == "step":
        state["x_in"], state["v_in"] = _pinned(sc.position), _pinned(sc.velocity)
        state["bodies"] = [(b, system.rigid_state(b)) for b, (_, rigid) in enumerate(sc.sample_boundaries) if rigid]
        if case["graph"]:
            system.set_step_graphs(case["graph"])
    if _restarts(case):
        ids = np.zeros(len(sc.position), np.uint32) if sc.fluid_id is None else sc.fluid_id
        state["checkpoint"] = {"fluid_id": ids, "position": sc.position, "velocity": sc.velocity, "mass": sc.mass,
                               "time_steps_propagated": 0, "current_time": 0.0}
    return state


def _restarts(case):
    """Cases that start each pass from a checkpoint: predicted integrator
    slots, bodies and CFL time steps all begin anew with it."""
    return case["kind"] == "ball" or case.get("scene") == "tank"


# ---- one pass --------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "server":
        return _run_server(state)
    system = state["system"]
    if case["kind"] == "plane":
        return system.get_quantity_at_positions(QUANTITIES[case["quantity"]], state["points"])
    if case["kind"] == "surface":
        return _fill(state, system.reconstruct_surfaces())
    if _restarts(case):
        for b, start in state.get("bodies", ()):
            system.set_rigid_state(b, start)
        system.continue_from_checkpoint(state["checkpoint"])
        system.step_host(case["steps"], None, None, state["x_out"], state["v_out"])
    else:
        system.step_host(case["steps"], state["x_in"], state["v_in"], state["x_out"], state["v_out"])
    if case["precision"] == "f64":
        return {"position": state["x_out"], "velocity": state["v_out"]}
    # f32 state: the program keeps its frame in f32, like the engine
    out = {"position": state["x"].copy_(state["x_out"]), "velocity": state["v"].copy_(state["v_out"])}
    if state.get("bodies"):
        out["bodies"] = np.stack([system.rigid_state(b) for b, _ in state["bodies"]]).astype(np.float32)
    return out


def _fill(state, meshes):
    """One fluid's mesh in the renderer's buffers, zeros behind it."""
    (_, vertices, indices), = meshes
    for buffer, values in ((state["vertices"], vertices), (state["indices"], indices)):
        buffer[:len(values)] = values
        buffer[len(values):] = 0
    return {"vertices": state["vertices"], "indices": state["indices"], "count": len(indices)}


def _run_server(state):
    server, out = state["server"], []
    tickets = [server.submit(sc, state["case"]["steps"], keep_state=True) for sc in state["scenes"]]
    for t, sc in zip(tickets, state["scenes"]):
        server.wait(t)
        x, v = server.fetch_state(t, len(sc.position))
        server.release(t)
        out.append({"position": x.astype(np.float32), "velocity": v.astype(np.float32)})
    return out


# ---- work ----------------------------------------------------------------------
_PAIRS = 32  # neighbors of a particle at a support of two spacings


def _particles(case):
    if case["kind"] == "ball":
        return 2.0 / 3.0 * math.pi * case["side"] ** 3
    if case["kind"] == "step" and case["scene"] == "tank":
        return 1.5 * 0.375 * case["side"] ** 3
    return float(case["side"]) ** 3


def _step_work(n, solver, word, steps):
    """State streams and pair arithmetic of `steps` updates (three sweeps of
    the implicit solvers, their least)."""
    pair_flops = {"SESPH": 60, "SESPHwSplitting": 100, "IISPH": 100 + 3 * 40, "IISPHwOST": 140 + 7 * 40}[solver]
    stream = {"SESPH": 40, "SESPHwSplitting": 60, "IISPH": 100 + 3 * 28, "IISPHwOST": 140 + 7 * 28}[solver]
    return steps * n * stream * word, steps * n * _PAIRS * pair_flops


def work(case):
    if case["kind"] == "server":
        sizes = np.exp(np.linspace(math.log(case["small"]), math.log(case["large"]), case["scenes"]))
        parts = [_step_work(float(n), "SESPH" if k % 2 == 0 else "IISPH", 4, case["steps"] + 1)
                 for k, n in enumerate(sizes)]
        return {"bytes": sum(b for b, _ in parts) + 100.0 * float(sizes.sum()), "flops": sum(f for _, f in parts)}
    n = _particles(case)
    if case["kind"] == "plane":
        points = case["rows"] * case["cols"]
        return {"bytes": 16.0 * points + 32.0 * n, "flops": points * _PAIRS * 30.0}
    if case["kind"] == "surface":
        # a lattice point per 0.375 spacings, and the mesh over the block's faces
        points = n / 0.375 ** 3
        faces = 6 * (case["side"] / 0.375) ** 2
        return {"bytes": 32.0 * n + 8.0 * points + 72.0 * faces, "flops": (points + n) * _PAIRS * 20.0}
    word = 8 if case["precision"] == "f64" else 4
    b, f = _step_work(n, case.get("solver", "IISPHwOST"), word, case["steps"] + (1 if _restarts(case) else 0))
    return {"bytes": b + 96.0 * n, "flops": f}


# ---- the same update in 64 bits ----------------------------------------------------
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(DEV, dtype)


def _pairs(a, b, h, drop_self=False):
    """(i, j) of all pairs with |a_i - b_j| < h."""
    lo = torch.minimum(a.amin(0), b.amin(0))
    ca, cb = torch.floor((a - lo) / h).long() + 1, torch.floor((b - lo) / h).long() + 1
    dims = torch.maximum(ca.amax(0), cb.amax(0)) + 2
    strides = torch.stack([torch.ones_like(dims[0]), dims[0], dims[0] * dims[1]])
    ka, kb = (ca * strides).sum(1), (cb * strides).sum(1)
    kb, order = torch.sort(kb)
    count = torch.bincount(kb, minlength=int(dims.prod()))
    start = torch.cumsum(count, 0) - count
    index = torch.arange(len(a), device=DEV)
    found = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = ka + dx + dy * strides[1] + dz * strides[2]
                c = count[k]
                i = torch.repeat_interleave(index, c)
                first = torch.cumsum(c, 0) - c
                j = order[start[k][i] + torch.arange(len(i), device=DEV) - first[i]]
                keep = (a[i] - b[j]).norm(dim=1) < h
                if drop_self:
                    keep &= i != j
                found.append((i[keep], j[keep]))
    return torch.cat([p for p, _ in found]), torch.cat([q for _, q in found])


def _kernel(r2, h):
    """W and the factor f of gradW = f r (cubic spline, support radius h)."""
    r = torch.sqrt(r2)
    q = r / h
    a, b = torch.clamp(1 - q, min=0), torch.clamp(0.5 - q, min=0)
    alpha = 16.0 / math.pi
    w = alpha / h ** 3 * (a ** 3 - 4 * b ** 3)
    f = alpha / h ** 4 * (12 * b ** 2 - 3 * a ** 2) / r
    return w, torch.where(r > 0, f, torch.zeros_like(f))


def _serendipity(field, p):
    """Cubic serendipity interpolant of a node lattice at p (NaN where the
    lattice has no value)."""
    xmin, xmax, n = _t(field.x_min), _t(field.x_max), _t(field.n, torch.long)
    nodes = _t(field.nodes)
    inside = ((p >= xmin) & (p <= xmax)).all(1)
    c = torch.minimum(torch.floor((p - xmin) / field.dx).long(), n - 1)
    c = torch.where(inside[:, None], c, torch.zeros_like(c))
    u = 2 * (p - (xmin + c.double() * field.dx)) / field.dx - 1
    nx, ny = 3 * int(n[0]) + 1, 3 * int(n[1]) + 1
    total = torch.zeros(len(p), dtype=torch.float64, device=DEV)

    def add(node, weight):
        off = [int(round((v + 1) * 1.5)) for v in node]
        at = ((3 * c[:, 2] + off[2]) * ny + 3 * c[:, 1] + off[1]) * nx + 3 * c[:, 0] + off[0]
        return total + nodes[at] * weight

    lin = {s: 1 + s * u for s in (-1.0, 1.0)}
    r2 = (u * u).sum(1)
    for x in (-1.0, 1.0):
        for y in (-1.0, 1.0):
            for z in (-1.0, 1.0):
                total = add((x, y, z), lin[x][:, 0] * lin[y][:, 1] * lin[z][:, 2] * (9 * r2 - 19) / 64)
    for d in range(3):
        e, g = [k for k in range(3) if k != d]
        for t in (-1.0 / 3.0, 1.0 / 3.0):
            for s0 in (-1.0, 1.0):
                for s1 in (-1.0, 1.0):
                    node = [0.0, 0.0, 0.0]
                    node[d], node[e], node[g] = t, s0, s1
                    total = add(node, 9.0 / 64.0 * (1 - u[:, d] ** 2) * (1 + 9 * u[:, d] * t) * lin[s0][:, e] * lin[s1][:, g])
    return torch.where(inside, total, torch.full_like(total, math.nan))


class _Exact:
    """System::update of a scene with static boundaries, on pair lists."""

    def __init__(self, sc, fields):
        p = sc.parameters
        self.sc, self.p, self.fields = sc, p, fields
        self.h, self.sp = p["kernel_support_radius"], p["rest_density_grid_spacing"]
        self.V0 = self.sp ** 3
        self.solver = sc.procedures["pressure_solver"]
        self.gamma = p["boundary_pressure_acceleration_weighting"]
        self.x, self.v, self.m = _t(sc.position), _t(sc.velocity), _t(sc.mass)
        if sc.sample_boundaries:
            self.xs = _t(_f32(np.concatenate([b for b, _ in sc.sample_boundaries])))
            i, j = _pairs(self.xs, self.xs, self.h)
            w, _ = _kernel(((self.xs[i] - self.xs[j]) ** 2).sum(1), self.h)
            total = torch.zeros(len(self.xs), dtype=torch.float64, device=DEV).index_add_(0, i, w)
            self.Vs = p["boundary_rest_volume_weighting"] / total
        self.dt = 0.0 if sc.cfl_time_step else p["time_increment"]
        self.update()

    def sum(self, i, values):
        shape = (len(self.x),) + values.shape[1:]
        return torch.zeros(shape, dtype=torch.float64, device=DEV).index_add_(0, i, values)

    def normal_samples(self, x):
        """(particle, sample position, sample volume) of the boundary neighbors of x."""
        if self.sc.sample_boundaries:
            i, s = _pairs(x, self.xs, self.h)
            return i, self.xs[s], self.Vs[s]
        sdf, vm = self.fields
        sd = _serendipity(sdf, x)
        g, e = [], sdf.dx / 6
        for d in range(3):
            step = torch.zeros(3, dtype=torch.float64, device=DEV)
            step[d] = e
            g.append((_serendipity(sdf, x + step) - _serendipity(sdf, x - step)) / (2 * e))
        g = torch.stack(g, 1)
        norm, vol = g.norm(dim=1), _serendipity(vm, x)
        i = torch.nonzero((sd < self.h) & (norm > 0.5) & (norm < 2) & (vol > 0))[:, 0]
        off = torch.clamp(sd[i] + 0.25 * self.sp, min=self.sp)
        xb = x[i] - g[i] / norm[i, None] * off[:, None]
        return i, xb, torch.clamp(vol[i], max=4.0 / 3.0 * math.pi * self.h ** 3)

    def viscous_samples(self, i, xb, Vb):
        if self.sc.sample_boundaries:
            return i, xb, Vb
        u = xb - self.x[i]
        helper = torch.where((u[:, :1] / u.norm(dim=1, keepdim=True)).abs() > 0.9,
                             _t([[0.0, 1.0, 0.0]]), _t([[1.0, 0.0, 0.0]]))
        t1 = torch.linalg.cross(u, helper)
        t2 = torch.linalg.cross(u, t1)
        t1, t2 = (0.5 * self.h * t / t.norm(dim=1, keepdim=True) for t in (t1, t2))
        return i.repeat(4), torch.cat([xb + t1, xb - t1, xb + t2, xb - t2]), 0.25 * Vb.repeat(4)

    def update(self):
        h, x, v, m = self.h, self.x, self.v, self.m
        if self.sc.cfl_time_step:
            speed = float(v.norm(dim=1).max())
            limit = self.p["cfl_number"] * self.sp / speed if speed > 0 else math.inf
            self.dt = min(self.p["max_time_increment"], limit)
        dt = self.dt
        i, j = self.i, self.j = _pairs(x, x, h, drop_self=True)
        r = x[i] - x[j]
        r2 = (r * r).sum(1)
        w, f = _kernel(r2, h)
        self.grad = f[:, None] * r
        b, xb, Vb = self.normal_samples(x)
        rb = x[b] - xb
        wb, fb = _kernel((rb * rb).sum(1), h)
        bW = self.sum(b, Vb * wb)
        self.bG = self.sum(b, (Vb * fb)[:, None] * rb)
        w0 = 0.5 * 16.0 / math.pi / h ** 3
        V = self.V = self.V0 / (self.V0 * (w0 + self.sum(i, w)) + bW)
        # gravity and viscosity
        a = torch.zeros_like(x)
        a[:, 2] = -G
        eps = 0.01 * self.sp ** 2
        visc = 10 * self.p["fluid_viscosity"] * V[j] * ((v[i] - v[j]) * r).sum(1) / (r2 + eps)
        a += self.sum(i, visc[:, None] * self.grad)
        c, xc, Vc = self.viscous_samples(b, xb, Vb)
        rc = x[c] - xc
        rc2 = (rc * rc).sum(1)
        inside = rc2 < h * h
        _, fc = _kernel(rc2, h)
        visc = 10 * self.p["boundary_viscosity"] * Vc * (v[c] * rc).sum(1) / (rc2 + eps) * torch.where(inside, fc, 0 * fc)
        a += self.sum(c, visc[:, None] * rc)
        if self.solver == "SESPH":
            self.pressure = self.p["stiffness"] * torch.clamp(self.V0 / V - 1, min=0)
            self.a = a + self.pressure_acceleration()
            return
        vs = v + dt * a
        if self.solver == "SESPHwSplitting":
            bGu = self.sum(b, fb[:, None] * rb)
            rho = m * w0 + self.sum(i, m[j] * w + dt * ((vs[i] - vs[j]) * self.grad).sum(1))
            rho += bW * m / self.V0 + dt * (vs * bGu).sum(1)
            self.pressure = self.p["stiffness"] * torch.clamp(self.V0 * rho / m - 1, min=0)
            self.a = a + self.pressure_acceleration()
        elif self.solver == "IISPH":
            self.solve(vs, True, None)
            self.a = a + self.pressure_acceleration()
        else:
            self.solve(vs, False, 4)
            vs = vs + dt * self.pressure_acceleration()
            self.solve(vs, True, None)
            a = self.pressure_acceleration()
            self.x_next, self.v_next = x + dt * vs + dt * dt * a, vs + dt * a

    def pressure_acceleration(self):
        i, j, V, p = self.i, self.j, self.V, self.pressure
        s = self.sum(i, (V[j] * (p[i] + p[j]))[:, None] * self.grad) + 2 * self.gamma * p[:, None] * self.bG
        return -(V / self.m)[:, None] * s

    def solve(self, vs, volume_source, sweeps):
        i, j, V, m, dt, bG = self.i, self.j, self.V, self.m, self.dt, self.bG
        S = self.sum(i, V[j, None] * self.grad)
        div = self.sum(i, V[j] * ((vs[i] - vs[j]) * self.grad).sum(1)) + (vs * bG).sum(1)
        s = (1 - self.V0 / V if volume_source else 0.0) - dt * div
        diag = -(V / m) * ((S + 2 * self.gamma * bG) * (S + bG)).sum(1)
        diag = dt * dt * (diag - V * self.sum(i, V[j] ** 2 / m[j] * (self.grad ** 2).sum(1)))
        omega, least = self.p["relaxation_factor"], self.p["min_diagonal_element"]
        self.pressure = torch.where(diag.abs() > least, torch.clamp(omega * s / diag, min=0), 0 * s)
        cap, done = self.p.get("max_solver_iterations", 0), 0
        while True:
            a = self.pressure_acceleration()
            A = dt * dt * (self.sum(i, V[j] * ((a[i] - a[j]) * self.grad).sum(1)) + (a * bG).sum(1))
            self.pressure = torch.where(diag < -least, torch.clamp(self.pressure + omega * (s - A) / diag, min=0),
                                        self.pressure)
            err = 100 * float(torch.where(s < 0, (A - s).abs(), 0 * s).mean())
            done += 1
            if sweeps is not None:
                if done >= sweeps:
                    return
            elif (done > 2 and err < self.p["target_density_error"]) or (cap and done >= cap):
                return

    def step(self):
        if self.solver == "IISPHwOST":
            self.x, self.v = self.x_next, self.v_next
        else:
            self.v = self.v + self.dt * self.a
            self.x = self.x + self.dt * self.v
        self.update()

    def quantity(self, points, quantity):
        q = _t(points)
        i, j = _pairs(q, self.x, self.h)
        zero = torch.zeros(len(q), dtype=torch.float64, device=DEV)
        w, _ = _kernel(((q[i] - self.x[j]) ** 2).sum(1), self.h)
        if quantity == "density":
            return zero.index_add(0, i, self.m[j] * w)
        if quantity == "speed":  # the container's samples are at rest
            vw = (self.V[j] * w)[:, None] * self.v[j]
            return torch.zeros_like(q).index_add(0, i, vw).norm(dim=1)
        b, xb, Vb = self.normal_samples(q)
        wb, _ = _kernel(((q[b] - xb) ** 2).sum(1), self.h)
        return self.V0 / (self.V0 * zero.index_add(0, i, w) + zero.index_add(0, b, Vb * wb))


def _stepped(sc, steps):
    e = _Exact(sc, _fields(sc))
    for _ in range(steps):
        e.step()
    return {"position": e.x.cpu(), "velocity": e.v.cpu()}


def exact(case, seed):
    if case["kind"] == "surface" or case.get("scene") == "tank":
        return None  # a mesh; bodies that move
    if case["kind"] == "server":
        if case["scenes"] * case["large"] * case["steps"] > 10_000_000:
            return None
        return [_stepped(sc, case["steps"]) for sc in _server_scenes(case, seed)]
    sc = _scene(case, seed)
    if case["kind"] == "plane":
        return _Exact(sc, _fields(sc)).quantity(_plane(case, sc, seed), case["quantity"])
    return _stepped(sc, case["steps"])
