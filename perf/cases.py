"""What the framework's users have it do, as cases that can be timed and compared.

A user of the solver advances smoke scenes (`Model.forward_step`), differentiates
rollouts (`simulate`, `jvp`, `vjp`) and runs or trains the warm-start network
(`WarmStartNetwork`).  Scenes, sizes and settings are those of the examples, the
tests and the benchmark:

  plume      walls, open top, inflow sphere: the benchmark's scene
  jets       the forward example's two pulsed jets, red-black sweeps, vorticity
  obstacles  the plume with a box and an ellipsoid in its way
  closed     the plume in a closed box (zero-gradient pressure: an anchor cell)
  periodic   periodic in x and z

`exact` restates every case in 64 bits with plain torch.  The fields of a case:

  work       forward, rollout, gradient, tangent, predict or train
  scene      see above (network cases: the scene of the training pairs)
  nx ny nz   the fluid grid, or the network's
  vorticity  vorticity confinement on
  sweeps     red-black Gauss-Seidel sweeps per solve; 0: Jacobi-PCG to 1e-6
  history    previous solutions that warm-start a solve; coarsening: factor of the
             coarse-grid correction; network: factor of the learned correction
             (0: none of each)
  steps      steps of a differentiated rollout; checkpoint: its interval (0: every
             state and cache is kept)
  batch      samples of a network call
"""
import math
import os

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WEIGHTS = os.path.join(ROOT, "diff_solver_b200", "weights", "warm_start_128.npz")
WARM_STEPS = 6  # steps a running simulation has behind it when a rollout case begins: its ring of solutions is full
DEVICE = "cuda"


def _case(name, work, scene, nx, ny, nz, **more):
    c = {"work": work, "scene": scene, "nx": nx, "ny": ny, "nz": nz, "vorticity": False, "sweeps": 0, "history": 0, "coarsening": 0,
         "network": 0, "steps": 1, "checkpoint": 0, "batch": 1}
    c.update(more)
    return {"name": name, **c} if name else c


def listed():
    return [
        # the default configuration's grid with its vorticity: interactive previews, where launches and latency count
        _case("forward_small_32x48x32", "forward", "plume", 32, 48, 32, vorticity=True),
        # the 64^3 plume by the plain solver: the benchmark's smallest configuration
        _case("forward_plume_64", "forward", "plume", 64, 64, 64),
        # a scene with colliders on a grid of no particular size, no power-of-two spacing
        _case("forward_obstacles_100x75x90", "forward", "obstacles", 100, 75, 90, vorticity=True),
        # the forward example as it ships: fixed red-black sweeps, vorticity, traces of several cells, metrics after the step
        _case("forward_jets_128x192x128", "forward", "jets", 128, 192, 128, vorticity=True, sweeps=160),
        # one step of a running simulation with the classical warm start, mid-sized
        _case("rollout_plume_128", "rollout", "plume", 128, 128, 128, history=5, coarsening=2),
        # the benchmark's headline: the running 256^3 plume with the learned correction
        _case("rollout_learned_256", "rollout", "plume", 256, 256, 256, history=5, coarsening=2, network=4),
        # the benchmark's large grid
        _case("rollout_large_512x512x256", "rollout", "plume", 512, 512, 256, history=5, coarsening=2),
        # the differentiable plume at its configured size, checkpointed, with the warm starts of both directions
        _case("gradient_plume_128", "gradient", "plume", 128, 128, 128, history=5, coarsening=2, steps=8, checkpoint=4),
        # a small inverse problem on a ragged grid with vorticity, the whole tape kept, plain solves
        _case("gradient_ragged_45x60x38", "gradient", "plume", 45, 60, 38, vorticity=True, steps=3),
        # a directional derivative along a short rollout
        _case("tangent_plume_64", "tangent", "plume", 64, 64, 64, steps=2),
        # the network as the headline runs it
        _case("predict_64", "predict", "plume", 64, 64, 64),
        # a training batch: loss and gradient of the energy loss
        _case("train_64_batch8", "train", "plume", 64, 64, 64, batch=8),
    ]


def _spread(rng, low, high, multiple=1):
    """A size between low and high, spread over its logarithm."""
    return max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high))) / multiple)) * multiple)


def draw(rng):
    work = rng.choice(["forward", "forward", "forward", "rollout", "rollout", "gradient", "gradient", "tangent", "predict", "train"])
    if work in ("predict", "train"):
        return _case(None, work, "plume", rng.choice([64, 128]), rng.choice([64, 128]), 16 * rng.randint(2, 8),
                     batch=1 if work == "predict" else rng.randint(1, 4))
    scenes = {"forward": ["plume", "plume", "jets", "obstacles", "closed", "periodic"], "rollout": ["plume", "plume", "closed", "periodic"],
              "gradient": ["plume", "periodic"], "tangent": ["plume", "periodic"]}
    scene = rng.choice(scenes[work])
    top = {"forward": 160, "rollout": 224, "gradient": 96, "tangent": 96}[work]
    if work == "rollout":  # the coarse grid divides the fine one
        f = rng.choice([2, 2, 4])
        nx, ny, nz = (_spread(rng, 48, top, f) for _ in range(3))
        return _case(None, work, scene, nx, ny, nz, history=rng.randint(3, 5), coarsening=f)
    nx, ny, nz = (_spread(rng, 24, top) for _ in range(3))
    vorticity = scene == "jets" or rng.random() < 0.4
    if work == "forward":
        return _case(None, work, scene, nx, ny, nz, vorticity=vorticity, sweeps=rng.randint(60, 160) if scene == "jets" else 0)
    steps = rng.randint(2, 5)
    return _case(None, work, scene, nx, ny, nz, vorticity=vorticity, steps=steps, checkpoint=rng.choice([0, 2]) if work == "gradient" else 0)


# ------------------------------------------------------------------ scenes
FIXED, ZERO_GRADIENT, NORMAL_FIXED, PERIODIC = 0, 1, 2, 3  # velocity faces; scalar faces: 0, 1, and 2 for periodic


def _scene(c):
    """Boundary modes (faces x-, x+, y-, y+, z-, z+; fixed values are 0),
    spacing, inflows, colliders, parameters and the size of the velocity."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    scene = c["scene"]
    h, walls = 1.0 / nx, NORMAL_FIXED
    s = {"h": h, "dt": 128.0 / 120.0 * h if scene == "jets" else 0.5 * h,  # the example: 1/120 at 1/128
         "velocity": [walls, walls, walls, ZERO_GRADIENT, walls, walls],
         "pressure": [1, 1, 1, 0, 1, 1], "scalar": [1, 1, 1, 0, 1, 1],
         "inflows": [(0.5, 0.1, 0.5 * nz / nx, 0.08, 1.0, 1.0)], "colliders": [], "speed": 0.1,
         "parameters": (0.0, -0.1, 0.5, 2.0 if c["vorticity"] else 0.0)}
    if scene == "jets":
        s.update(inflows=[], speed=1.0, parameters=(0.0, -0.1, 1.0, 2.0))
    if scene == "closed":
        s["velocity"][3] = walls
        s["pressure"] = [1] * 6
        s["scalar"] = [1] * 6
    if scene == "periodic":
        s["velocity"] = [PERIODIC, PERIODIC, walls, ZERO_GRADIENT, PERIODIC, PERIODIC]
        s["pressure"] = [2, 2, 1, 0, 2, 2]
        s["scalar"] = [2, 2, 1, 1, 2, 2]
    if scene == "obstacles":
        ly, lz = ny / nx, nz / nx
        s["colliders"] = [("box", (0.55, 0.45 * ly, 0.5 * lz), (0.12, 0.08 * ly, 0.1 * lz), (0.05, 0.0, 0.02), 0.5, 0.25),
                          ("ellipsoid", (0.3, 0.7 * ly, 0.35 * lz), (0.15, 0.1 * ly, 0.12 * lz), (-0.02, 0.0, 0.05), 0.2, 0.7)]
    return s


def _configuration(c):
    from diff_solver_b200 import data as D
    s = _scene(c)
    if c["scene"] == "jets":
        from diff_solver_b200.simulation import make_configuration
        cfg = make_configuration(_jet_options(c))
    else:
        cfg = D.Configuration(resolution=[c["nx"], c["ny"], c["nz"]], cell_size=s["h"], time_step=s["dt"])
        for f, m in zip(cfg.velocity_boundary.faces(), s["velocity"]):
            f.mode = D.VelocityBoundaryMode(m)
        for b, modes in ((cfg.pressure_boundary, s["pressure"]), (cfg.density_boundary, s["scalar"]), (cfg.temperature_boundary, s["scalar"])):
            for f, m in zip(b.faces(), modes):
                f.mode = D.ScalarBoundaryMode(m)
        cfg.inflows = [D.Inflow(D.Vector3(*v[:3]), *v[3:]) for v in s["inflows"]]
        for kind, centre, size, velocity, density, temperature in s["colliders"]:
            shape = (D.Box if kind == "box" else D.Ellipsoid)(D.Vector3(*centre), D.Vector3(*size))
            cfg.colliders.append(D.Collider(shape, D.Vector3(*velocity), density, temperature))
        cfg.pressure_max_iterations = 20000
    cfg.vorticity_confinement_enabled = c["vorticity"]
    cfg.warm_start_history = c["history"]
    cfg.warm_start_coarsening = c["coarsening"]
    return cfg


def _jet_options(c):
    from diff_solver_b200.simulation import ForwardSimulationOptions
    s = _scene(c)
    return ForwardSimulationOptions(resolution=(c["nx"], c["ny"], c["nz"]), cell_size=s["h"], time_step=s["dt"], pressure_iterations=c["sweeps"])


JET_STEP = 30  # the step whose controls the jets case writes


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cpu").manual_seed(int(seed) % (1 << 31))


def _edges(n, count, wave, dev):
    """count sines over n + 1 edges, zero at both ends."""
    t = torch.arange(n + 1, dtype=torch.float64, device=dev) / n
    return torch.sin(math.pi * wave.to(dev)[:count, None] * t[None])


def _inputs(c, seed, dev):
    """The fluid state and the controls of a case, FP32: smoke puffs, a smooth
    velocity without divergence that vanishes at the walls (the discrete curl
    of a vector potential on the edges), as a projected plume has."""
    s, g = _scene(c), _generator(seed)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    h, modes = s["h"], 8
    size = torch.tensor([nx, ny, nz], dtype=torch.float64) * h
    wave = torch.randint(1, 4, (3, 3, modes), generator=g).double() * 2.0
    amp = torch.randn((3, modes), generator=g, dtype=torch.float64)

    def centres(n):
        return (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n

    def potential(axis):
        """Component `axis` of the potential: cell centres along its own axis, edges along the other two."""
        parts = []
        for d, n in enumerate((nx, ny, nz)):
            parts.append(torch.cos(math.pi * wave[axis, d].to(dev)[:, None] * centres(n)[None]) if d == axis else _edges(n, modes, wave[axis, d], dev))
        return torch.einsum("mk,mj,mi->kji", parts[2] * amp[axis].to(dev)[:, None], parts[1], parts[0])

    px, py, pz = (potential(a) for a in range(3))
    u = [pz.diff(dim=1) - py.diff(dim=0), px.diff(dim=0) - pz.diff(dim=2), py.diff(dim=2) - px.diff(dim=1)]
    scale = s["speed"] / max(float(v.abs().max()) for v in u)
    velocity = [(v * scale).float().contiguous() for v in u]
    x, y, z = (centres(n) * float(size[d]) for d, n in enumerate((nx, ny, nz)))

    def puffs(count, height):
        out = torch.zeros((nz, ny, nx), dtype=torch.float64, device=dev)
        r = torch.rand((count, 4), generator=g, dtype=torch.float64)
        for k in range(count):
            c0 = [float(size[0]) * (0.35 + 0.3 * float(r[k, 0])), float(size[1]) * (0.08 + 0.5 * float(r[k, 1])),
                  float(size[2]) * (0.35 + 0.3 * float(r[k, 2]))]
            w = float(size.min()) * (0.06 + 0.08 * float(r[k, 3]))
            e = [torch.exp(-0.5 * ((v - m) / w) ** 2) for v, m in zip((x, y, z), c0)]
            out += torch.einsum("k,j,i->kji", e[2], e[1], e[0])
        return (out.clamp(max=1.0) * height).float()

    state = [puffs(4, 1.0), puffs(4, 1.0), *velocity]
    if c["work"] in ("rollout",) or (c["work"] == "forward" and c["scene"] == "plume"):
        control = [torch.zeros((nz, ny, nx), dtype=torch.float32, device=dev) for _ in range(5)]
    else:  # a user's sources and forces
        control = [puffs(2, 0.5), puffs(2, 0.5), puffs(2, 0.2), puffs(2, 0.2), puffs(2, -0.2)]
    return state, control


def _seeds(c, seed, dev):
    """A loss gradient at the last state (density and velocity), or an initial tangent."""
    state, _ = _inputs(dict(c, work="seed"), seed + 7919, dev)
    return state


def _pairs(c, seed, dev):
    """Training pairs on the network grid: smooth pressures and their right-hand sides."""
    out = []
    for b in range(c["batch"]):
        (rho, temp, *_), _ = _inputs(c, seed * 64 + b, dev)
        out.append(rho.double() - temp.double())
    p = torch.stack(out)
    rhs = torch.stack([_Grid(c, dev).laplacian(v) for v in p])
    noise = torch.randn(rhs.shape, generator=torch.Generator(device=dev).manual_seed(seed % (1 << 31)), device=dev, dtype=torch.float32)
    rhs = rhs.float() + 0.05 * float(rhs.std()) * noise
    return rhs.contiguous(), p.float().contiguous()


# ------------------------------------------------------------------ cases
class _State:
    pass


def prepare(c, seed):
    dev = torch.device(DEVICE)
    t = _State()
    t.case = c
    if c["work"] in ("predict", "train"):
        from diff_solver_b200.model import scalar_boundary
        from diff_solver_b200.warm_start import WarmStartNetwork
        t.net = WarmStartNetwork((c["nx"], c["ny"], c["nz"]), max_batch=c["batch"])
        t.net.load(WEIGHTS)
        if c["work"] == "train":
            t.net.set_loss("energy", scalar_boundary(_configuration(c).pressure_boundary))
        t.rhs, t.pressure = (v.reshape(c["batch"], -1) for v in _pairs(c, seed, dev))
        return t
    from diff_solver_b200.model import ExecutionMode, Model, fill_parameters, tensors_of
    t.model = m = Model(_configuration(c))
    mode = ExecutionMode.differentiable if c["work"] in ("gradient", "tangent") else ExecutionMode.forward
    t.ctx = ctx = m.allocate_context(mode)
    if c["network"]:
        from diff_solver_b200.warm_start import WarmStartNetwork
        f = c["network"]
        t.net = WarmStartNetwork((c["nx"] // f, c["ny"] // f, c["nz"] // f), factor=f)
        t.net.load(WEIGHTS)
        ctx.set_learned_warm_start(t.net)
    state, control = _inputs(c, seed, dev)

    def fill(target, values):
        for a, b in zip(tensors_of(target), values):
            a.copy_(b.reshape(-1))
        return target

    t.state = fill(m.allocate_state(ctx), state)
    t.control = fill(m.allocate_control(ctx), control)
    t.parameters = fill_parameters(m.allocate_parameters(ctx), *_scene(c)["parameters"])
    if c["work"] in ("forward", "rollout"):
        t.next = m.allocate_state(ctx)
        t.cache = m.allocate_step_cache(ctx)
        t.metrics = torch.zeros(6, dtype=torch.float64, device=dev)
        if c["work"] == "rollout":
            for _ in range(WARM_STEPS):
                run(t)
    else:
        t.controls = [t.control] * c["steps"]
        seeds = _seeds(c, seed, dev)
        if c["work"] == "gradient":
            t.adjoint = fill(m.allocate_state_adjoint(ctx), seeds)
        else:
            t.tangent = fill(m.allocate_state_tangent(ctx), seeds)
            t.control_tangents = [t.control] * c["steps"]
            t.parameter_tangent = fill_parameters(m.allocate_parameter_tangent(ctx), 0.1, 0.2, -0.1, 0.3)
    return t


def run(t):
    from diff_solver_b200.model import tensors_of
    c = t.case
    if c["work"] == "predict":
        return t.net.predict(t.rhs)
    if c["work"] == "train":
        return t.net.gradient(t.rhs, t.pressure)
    if c["work"] == "forward":
        if c["scene"] == "jets":  # the example's step
            from diff_solver_b200.simulation import reduce_metrics, write_control
            write_control(t.ctx, t.control, JET_STEP, _jet_options(c))
        t.model.forward_step(t.state, t.control, t.parameters, t.next, t.cache, t.ctx)
        if c["scene"] == "jets":
            reduce_metrics(t.ctx, t.next, t.cache, t.metrics)
            return tensors_of(t.next) + [t.metrics]
        return tensors_of(t.next)
    if c["work"] == "rollout":  # the simulation moves on by one step
        t.model.forward_step(t.state, t.control, t.parameters, t.next, t.cache, t.ctx)
        t.state, t.next = t.next, t.state
        return tensors_of(t.state)
    from diff_solver_b200.solver import TapeMode, jvp, simulate, vjp
    if c["history"]:
        t.ctx.reset_warm_start()  # a new trajectory
    mode = TapeMode.checkpoint if c["checkpoint"] else TapeMode.store_all
    tape = simulate(t.model, t.ctx, t.state, t.controls, t.parameters, mode, c["checkpoint"])
    if c["work"] == "gradient":
        g = vjp(t.model, t.ctx, tape, t.controls, t.parameters, {c["steps"]: t.adjoint})
        return {"state": tensors_of(tape.states[-1]), "initial": tensors_of(g.initial_state), "controls": [tensors_of(v) for v in g.controls],
                "parameters": torch.cat(tensors_of(g.parameters))}
    tangents = jvp(t.model, t.ctx, tape, t.controls, t.parameters, t.tangent, t.control_tangents, t.parameter_tangent)
    return {"state": tensors_of(tape.states[-1]), "tangents": [tensors_of(v) for v in tangents[1:]]}


def work(c):
    """Unique bytes and rough operations.  A step reads its state and controls
    and writes its state and step cache (sourced fields, force, two face
    fields, with vorticity its 11 cell fields); an adjoint step reads the cache
    and writes 64-bit gradients of all its inputs; about 250 operations per
    face and 300 per cell of advection, half as many again for a tangent,
    three times as many for an adjoint."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    n = float(nx * ny * nz)
    if c["work"] in ("predict", "train"):
        layers = [(2, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (64, 64, 3), (64, 64, 3), (64, 32, 2), (32, 16, 1),
                  (16, 16, 0), (16, 1, 0)]
        flops = sum(2.0 * 27 * a * b * n * c["batch"] / 8 ** l for a, b, l in layers)
        weights = sum(27 * a * b for a, b, _ in layers)
        if c["work"] == "predict":
            return {"bytes": 8 * n + 2 * weights, "flops": flops}
        return {"bytes": 8 * n * c["batch"] + 6 * weights, "flops": 3 * flops}
    f = float((nx + 1) * ny * nz + nx * (ny + 1) * nz + nx * ny * (nz + 1))
    cache = 4 * (5 * n + 2 * f + (11 * n if c["vorticity"] else 0))
    step = 4 * (9 * n + 2 * f) + cache
    flops = 250 * f + 300 * n
    if c["work"] == "gradient":
        again = 2 if c["checkpoint"] else 1
        return {"bytes": c["steps"] * (again * step + cache + 8 * (9 * n + 2 * f)), "flops": c["steps"] * flops * (again + 3)}
    if c["work"] == "tangent":
        return {"bytes": c["steps"] * (step + cache + 4 * (9 * n + 2 * f)), "flops": c["steps"] * flops * 2.5}
    return {"bytes": step, "flops": flops}


def tolerance(c):
    """About four times what a step was seen to differ from `exact`."""
    if c["work"] == "predict":  # bf16 activations and weights: 4e-3
        return {"rel": 1.5e-2}
    if c["work"] == "train":  # and bf16 gradients: 2e-2 already
        return {"rel": 3e-2, "max": 0.9}
    # 32-bit fields, a pressure to a relative residual of 1e-6: 1e-6 in the fields, at single values up to 8e-4
    if c["work"] in ("forward", "rollout"):
        return {"rel": 1e-5 if c["scene"] == "obstacles" else 5e-6, "max": 5e-3}
    # derivatives of trilinear samples jump at the cells' edges, where a trace may end on either side
    # within its rounding: 2e-5 in tangents, up to 9e-3 in gradients, at single values as much as the value
    if c["work"] == "tangent":
        return {"rel": 1e-4, "max": 2e-2}
    return {"rel": 2e-2, "max": 0.9}


# ------------------------------------------------------------------ 64 bits
class _Grid:
    """The step of the smoke model in 64 bits on whole arrays [z, y, x]."""

    def __init__(self, c, dev):
        s = _scene(c)
        self.c, self.dev = c, dev
        self.n = (c["nx"], c["ny"], c["nz"])
        self.h, self.dt = float(np.float32(s["h"])), float(np.float32(s["dt"]))
        self.vm, self.pm, self.sm = s["velocity"], s["pressure"], s["scalar"]
        self.vper = [self.vm[2 * d] == PERIODIC and self.vm[2 * d + 1] == PERIODIC for d in range(3)]
        self.pper = [self.pm[2 * d] == 2 and self.pm[2 * d + 1] == 2 for d in range(3)]
        self.sper = [self.sm[2 * d] == 2 and self.sm[2 * d + 1] == 2 for d in range(3)]
        ix = [torch.arange(n, device=dev) for n in self.n]
        centre = [(v.float() + 0.5) * np.float32(s["h"]) for v in ix]  # the kernels test cell centres in 32 bits
        cx, cy, cz = centre[0][None, None], centre[1][None, :, None], centre[2][:, None, None]
        shape = self.n[::-1]
        self.hit = torch.zeros(shape, dtype=torch.bool, device=dev)
        for px, py, pz, r, _, _ in s["inflows"]:  # they all set 1
            a, b, d = (v - np.float32(p) for v, p in ((cx, px), (cy, py), (cz, pz)))
            self.hit |= a * a + b * b + d * d <= np.float32(r) * np.float32(r)
        self.solid = None
        if s["colliders"]:
            which = torch.full(shape, -1, dtype=torch.long, device=dev)
            for k, (kind, p, q, *_) in enumerate(s["colliders"]):
                d = [v - np.float32(m) for v, m in zip((cx, cy, cz), p)]
                if kind == "box":
                    inside = (d[0].abs() <= np.float32(q[0])) & (d[1].abs() <= np.float32(q[1])) & (d[2].abs() <= np.float32(q[2]))
                else:
                    e = [v / np.float32(w) for v, w in zip(d, q)]
                    inside = e[0] * e[0] + e[1] * e[1] + e[2] * e[2] <= 1.0
                which[inside.expand(shape)] = k
            self.solid = which >= 0
            table = [torch.tensor([float(np.float32(v)) for v in col] + [0.0], dtype=torch.float64, device=dev)
                     for col in zip(*[(*k[3], k[4], k[5]) for k in s["colliders"]])]
            self.solid_velocity, self.solid_scalar = [t[which] for t in table[:3]], [t[which] for t in table[3:]]
        self.fluid = None if self.solid is None else (~self.solid).double()
        free = not any(m == 0 for m in self.pm)
        self.anchor = None
        if free:
            self.anchor = 0 if self.solid is None else int((~self.solid).reshape(-1).nonzero()[0])

    def shape(self, axis):
        return tuple(self.n[d] + (axis == d) for d in range(3))

    # -------------------------------------------------- sampling
    def _load(self, v, axis, x, y, z):
        """v at integer coordinates: axis 0..2 a face component, -1 cells.
        Beyond a fixed face the value is 0; else the clamped or wrapped element."""
        size = self.shape(axis)
        per = self.sper if axis < 0 else self.vper
        fixed, at = None, []
        for d, q in enumerate((x, y, z)):
            low, high = q < 0, q >= size[d]
            if axis < 0:  # below the grid also counts as beyond its upper end
                const = [low] * (self.sm[2 * d] == 0) + [low | high] * (self.sm[2 * d + 1] == 0)
            else:
                const = [m for m, mode in ((low, self.vm[2 * d]), (high, self.vm[2 * d + 1])) if mode == FIXED or (mode == NORMAL_FIXED and axis == d)]
            for m in const:
                fixed = m if fixed is None else fixed | m
            at.append(q.remainder(self.n[d]) if per[d] else q.clamp(0, size[d] - 1))
        got = v.reshape(-1)[at[0] + size[0] * (at[1] + size[1] * at[2])]
        return got if fixed is None else torch.where(fixed, torch.zeros_like(got), got)

    def sample(self, v, axis, p):
        lower, weight = [], []
        for d in range(3):
            g = p[d] / self.h - (0.0 if axis == d else 0.5)
            f = g.detach().floor()
            lower.append(f.long())
            weight.append(g - f)
        total = 0.0
        for k in range(8):
            o = [k & 1, (k >> 1) & 1, k >> 2]
            w = 1.0
            for d in range(3):
                w = w * (weight[d] if o[d] else 1.0 - weight[d])
            total = total + w * self._load(v, axis, *(lower[d] + o[d] for d in range(3)))
        return total

    def _solid_at(self, p):
        at = []
        for d in range(3):
            q = p[d]
            if self.vper[d]:
                q = q - (q / (self.n[d] * self.h)).floor() * self.n[d] * self.h
            i = (q / self.h).floor().long()
            at.append(torch.where((i < 0) | (i >= self.n[d]), self.n[d] - 1, i))  # as unsigned numbers clamp
        return self.solid.reshape(-1)[at[0] + self.n[0] * (at[1] + self.n[1] * at[2])]

    def trace(self, u, s):
        v0 = [self.sample(u[a], a, s) for a in range(3)]
        mid = [s[d] - 0.5 * self.dt * v0[d] for d in range(3)]
        v1 = [self.sample(u[a], a, mid) for a in range(3)]
        end = [s[d] - self.dt * v1[d] if self.vper[d] else (s[d] - self.dt * v1[d]).clamp(0.0, self.n[d] * self.h) for d in range(3)]
        if self.solid is None:
            return end
        inside = self._solid_at([e.detach() for e in end])
        lo, hi = torch.zeros_like(end[0]).detach(), torch.ones_like(end[0]).detach()
        for _ in range(8):
            f = 0.5 * (lo + hi)
            into = self._solid_at([s[d] + f * (end[d].detach() - s[d]) for d in range(3)])
            lo, hi = torch.where(into, lo, f), torch.where(into, f, hi)
        return [torch.where(inside, s[d] + lo * (end[d] - s[d]), end[d]) for d in range(3)]

    def _positions(self, axis, z0, z1):
        size = self.shape(axis)
        ax = [(torch.arange(size[d], device=self.dev).double() + (0.0 if axis == d else 0.5)) * self.h for d in range(3)]
        return [t.contiguous() for t in torch.broadcast_tensors(ax[0][None, None], ax[1][None, :, None], ax[2][z0:z1, None, None])]

    def _advect(self, axis, u, fields):
        """fields (of component `axis`, or cells) at the traces' ends, in slabs of a few million values."""
        size = self.shape(axis)
        slab = max(1, 4_000_000 // (size[0] * size[1]))
        out = [[] for _ in fields]
        for z0 in range(0, size[2], slab):
            end = self.trace(u, self._positions(axis, z0, min(size[2], z0 + slab)))
            for k, v in enumerate(fields):
                out[k].append(self.sample(v, axis, end))
        return [torch.cat(o) for o in out]

    # -------------------------------------------------- faces and cells
    def _beside(self, axis, v):
        """v of the lower and of the upper cell beside each face of a component, zero outside the grid."""
        dim = 2 - axis
        pad = torch.zeros_like(v.narrow(dim, 0, 1))
        return torch.cat([pad, v], dim), torch.cat([v, pad], dim)

    def _force_on_faces(self, axis, f):
        one = torch.ones_like(f) if self.solid is None else self.fluid
        lo, hi = self._beside(axis, f * one)
        a, b = self._beside(axis, one)
        return (lo + hi) / (a + b).clamp(min=1.0)

    def _difference(self, v, axis):
        """v(c + 1) - v(c - 1) along an axis; past either end the last cell is read."""
        dim = 2 - axis
        last = v.narrow(dim, self.n[axis] - 1, 1)
        up = torch.cat([v.narrow(dim, 1, self.n[axis] - 1), last], dim)
        down = torch.cat([last, v.narrow(dim, 0, self.n[axis] - 1)], dim)
        return up - down

    def _vorticity_force(self, u, strength):
        eps = float(np.float32(1e-6))
        one = 1.0 if self.solid is None else self.fluid
        centred = [one * 0.5 * (u[a].narrow(2 - a, 0, self.n[a]) + u[a].narrow(2 - a, 1, self.n[a])) for a in range(3)]
        k = 0.5 / self.h
        d = self._difference
        w = [one * k * (d(centred[2], 1) - d(centred[1], 2)), one * k * (d(centred[0], 2) - d(centred[2], 0)),
             one * k * (d(centred[1], 0) - d(centred[0], 1))]
        mag = torch.sqrt(w[0] ** 2 + w[1] ** 2 + w[2] ** 2 + eps * eps)
        g = [one * k * d(mag, a) for a in range(3)]
        length = torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2 + eps * eps)
        m = [v / length for v in g]
        s = strength * self.h
        return [s * (m[1] * w[2] - m[2] * w[1]), s * (m[2] * w[0] - m[0] * w[2]), s * (m[0] * w[1] - m[1] * w[0])]

    # -------------------------------------------------- pressure
    def _neighbours(self, p):
        """The sum over a cell's connected neighbours, and what the cell's own value is multiplied by."""
        total, count = torch.zeros_like(p), torch.zeros_like(p)
        one = torch.ones_like(p) if self.solid is None else self.fluid
        for d in range(3):
            dim, n = 2 - d, self.n[d]
            for side in (0, 1):
                if self.pper[d]:
                    nb, there = (torch.roll(v, -1 if side else 1, dim) for v in (p * one, one))
                else:
                    pad = torch.zeros_like(p.narrow(dim, 0, 1))
                    edge = pad + (1.0 if self.pm[2 * d + side] == 0 else 0.0)
                    part = [v.narrow(dim, 1, n - 1) if side else v.narrow(dim, 0, n - 1) for v in (p * one, one)]
                    nb, there = (torch.cat([v, e] if side else [e, v], dim) for v, e in zip(part, (pad, edge)))
                total, count = total + nb, count + there
        return total, count

    def laplacian(self, p):
        total, count = self._neighbours(p)
        return count * p - total

    def _modes(self):
        """Eigenbases and eigenvalues of the operator along each axis."""
        if not hasattr(self, "basis"):
            self.basis = []
            for d, n in enumerate(self.n):
                t = torch.diag(torch.full((n,), 2.0, dtype=torch.float64)) - torch.diag(torch.ones(n - 1, dtype=torch.float64), 1) - \
                    torch.diag(torch.ones(n - 1, dtype=torch.float64), -1)
                if self.pper[d]:
                    t[0, -1] -= 1.0
                    t[-1, 0] -= 1.0
                else:
                    t[0, 0] -= float(self.pm[2 * d] != 0)
                    t[-1, -1] -= float(self.pm[2 * d + 1] != 0)
                lam, q = torch.linalg.eigh(t)
                self.basis.append((lam.to(self.dev), q.to(self.dev)))
        return self.basis

    def solve(self, b):
        """A p = b: without colliders by the eigenbases, else by conjugate gradients to 1e-12."""
        if self.solid is not None:
            return self._conjugate_gradients(b)
        (lx, qx), (ly, qy), (lz, qz) = self._modes()
        if self.anchor is not None:  # the anchor is held at 0: its row takes up the sum of the others
            b = b.reshape(-1)
            rest = b[1:]
            b = torch.cat([-rest.sum()[None], rest]).reshape(self.n[::-1])
        b = torch.matmul(b, qx)
        b = torch.matmul(qy.T, b)
        b = torch.matmul(qz.T, b.reshape(self.n[2], -1)).reshape(self.n[::-1])
        lam = lx[None, None] + ly[None, :, None] + lz[:, None, None]
        inverse = 1.0 / lam
        if self.anchor is not None:
            inverse.reshape(-1)[0] = 0.0
        b = b * inverse
        b = torch.matmul(qz, b.reshape(self.n[2], -1)).reshape(self.n[::-1])
        p = torch.matmul(torch.matmul(qy, b), qx.T)
        return p if self.anchor is None else p - p[0, 0, 0]

    def _conjugate_gradients(self, b):
        _, count = self._neighbours(b)
        active = self.fluid * (count > 0)
        if self.anchor is not None:
            active.reshape(-1)[self.anchor] = 0.0
        inverse = active / count.clamp(min=1.0)
        b = b * active
        x, r = torch.zeros_like(b), b.clone()
        z = r * inverse
        p, rz, end = z, (r * z).sum(), 1e-24 * (b * b).sum()
        for k in range(20000):
            if k % 20 == 0 and bool((r * r).sum() <= end):
                break
            q = self.laplacian(p) * active
            a = rz / (p * q).sum()
            x, r = x + a * p, r - a * q
            z = r * inverse
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
        return x

    def sweeps(self, b, count):
        """That many red-black Gauss-Seidel sweeps from zero."""
        ix = [torch.arange(n, device=self.dev) for n in self.n]
        parity = (ix[0][None, None] + ix[1][None, :, None] + ix[2][:, None, None]) % 2
        p = torch.zeros_like(b)
        _, diag = self._neighbours(p)
        for _ in range(count):
            for colour in (0, 1):
                total, _ = self._neighbours(p)
                p = torch.where(parity == colour, (b + total) / diag, p)
        return p

    # -------------------------------------------------- the step
    def step(self, state, control, parameters):
        rho, temp, u = state[0], state[1], list(state[2:])
        ambient, beta_rho, beta_temp, strength = parameters
        one = 1.0 if self.solid is None else self.fluid
        rho, temp = (torch.where(self.hit, torch.ones_like(v), v + self.dt * s) * one for v, s in ((rho, control[0]), (temp, control[1])))
        force = [f * one for f in control[2:]]
        force[1] = force[1] + one * (beta_rho * rho + beta_temp * (temp - ambient))
        if self.c["vorticity"]:
            force = [f + v for f, v in zip(force, self._vorticity_force(u, strength))]
        u = [u[a] + self.dt * self._force_on_faces(a, force[a]) for a in range(3)]
        u = [self._constrain(a, self._advect(a, u, [u[a]])[0]) for a in range(3)]
        before = u
        div = sum(u[a].diff(dim=2 - a) for a in range(3)) / self.h
        b = -self.h * self.h * div / self.dt * one
        if self.anchor is not None:
            keep = torch.ones_like(b)
            keep.reshape(-1)[self.anchor] = 0.0
            b = b * keep
        p = self.sweeps(b, self.c["sweeps"]) if self.c["sweeps"] else self.solve(b)
        out = []
        for a in range(3):
            lo, hi = self._beside(a, p)
            both = torch.ones_like(p) if self.solid is None else self.fluid
            first, second = self._beside(a, both)
            out.append(u[a] - self.dt * (hi - lo) / self.h * first * second)
        u = out
        rho, temp = self._advect(-1, u, [rho, temp])
        if self.solid is not None:
            rho, temp = (torch.where(self.solid, s, v) for s, v in zip(self.solid_scalar, (rho, temp)))
        return [rho, temp, *u], before

    def _constrain(self, a, v):
        dim, n = 2 - a, self.n[a]
        if self.solid is not None:
            lo, hi = self._beside(a, self.solid.double())
            sl, sh = self._beside(a, self.solid_velocity[a])
            beside = lo + hi
            v = torch.where(beside > 0, (sl + sh) / beside.clamp(min=1.0), v)
        if self.vper[a]:
            return torch.cat([v.narrow(dim, 0, n), v.narrow(dim, 0, 1)], dim)
        first, last = v.narrow(dim, 0, 1), v.narrow(dim, n, 1)
        if self.vm[2 * a] in (FIXED, NORMAL_FIXED):
            first = torch.zeros_like(first)
        if self.vm[2 * a + 1] in (FIXED, NORMAL_FIXED):
            last = torch.zeros_like(last)
        return torch.cat([first, v.narrow(dim, 1, n - 1), last], dim)

    def metrics(self, state, before):
        """The example's metrics: mass, maxima of density, temperature and speed, squared divergences."""
        rho, temp, u = state[0], state[1], state[2:]
        speed = sum((0.5 * (v.narrow(2 - a, 0, self.n[a]) + v.narrow(2 - a, 1, self.n[a]))) ** 2 for a, v in enumerate(u)).sqrt()
        div = [sum(v.diff(dim=2 - a) for a, v in enumerate(w)) / self.h for w in (before, u)]
        return torch.stack([rho.sum(), rho.max().clamp(min=0), temp.max().clamp(min=0), speed.max(), (div[0] ** 2).sum(), (div[1] ** 2).sum()])


def _jet_control(c, dev):
    """The example's controls at JET_STEP: two Gaussian jets pulsing in antiphase."""
    s = _scene(c)
    f = lambda v: float(np.float32(v))  # noqa: E731  (the options are 32-bit numbers)
    x, y, z = ((torch.arange(n, device=dev).double() + 0.5) * f(s["h"]) for n in (c["nx"], c["ny"], c["nz"]))
    phase = 2.0 * math.pi * JET_STEP * f(s["dt"]) / f(0.9)
    jets = []
    for centre, shift in (((0.25, 0.10, 0.36), 0.0), ((0.75, 0.10, 0.64), math.pi)):
        e = [torch.exp(-0.5 * ((v - f(m)) / f(0.055)) ** 2) for v, m in zip((x, y, z), centre)]
        jets.append((0.75 + 0.25 * math.sin(phase + shift)) * torch.einsum("k,j,i->kji", e[2], e[1], e[0]))
    left, right = jets
    push = [left * f(p) + right * f(q) for p, q in zip((3.5, 5.0, 1.8), (-3.5, 5.0, -1.8))]
    return [4.0 * (left + right), 8.0 * (left + right), *push]


def _exact_fluid(c, seed):
    dev = torch.device(DEVICE if torch.cuda.is_available() else "cpu")
    g = _Grid(c, dev)
    state, control = _inputs(c, seed, dev)
    state, control = [v.double() for v in state], [v.double() for v in control]
    if c["scene"] == "jets":
        control = _jet_control(c, dev)
    parameters = [torch.tensor(float(np.float32(v)), dtype=torch.float64, device=dev) for v in _scene(c)["parameters"]]
    flat = lambda vs: [v.reshape(-1) for v in vs]  # noqa: E731
    if c["work"] in ("forward", "rollout"):
        with torch.no_grad():
            for _ in range(WARM_STEPS + 1 if c["work"] == "rollout" else 1):
                state, before = g.step(state, control, parameters)
            return flat(state) + ([g.metrics(state, before)] if c["scene"] == "jets" else [])
    seeds = [v.double() for v in _seeds(c, seed, dev)]
    if c["work"] == "tangent":
        primal, tangent = [*state, *control, *parameters], None
        rates = [torch.tensor(float(np.float32(v)), dtype=torch.float64, device=dev) for v in (0.1, 0.2, -0.1, 0.3)]
        out = []
        tangent = seeds
        for _ in range(c["steps"]):
            def one(*v):
                return tuple(g.step(list(v[:5]), list(v[5:10]), list(v[10:]))[0])
            state, tangent = torch.func.jvp(one, (*state, *control, *parameters), (*tangent, *control, *rates))
            out.append(flat(tangent))
        return {"state": flat(state), "tangents": out}
    from torch.utils.checkpoint import checkpoint
    first = [v.requires_grad_() for v in state]
    controls = [[v.clone().requires_grad_() for v in control] for _ in range(c["steps"])]
    parameters = [v.requires_grad_() for v in parameters]
    state = first
    for k in range(c["steps"]):
        state = checkpoint(lambda s, q, w: g.step(s, q, w)[0], state, controls[k], parameters, use_reentrant=False)
    wanted = [*first, *[v for q in controls for v in q], *parameters]
    got = torch.autograd.grad(state, wanted, seeds, allow_unused=True)
    got = [torch.zeros_like(w) if v is None else v for v, w in zip(got, wanted)]
    split = [flat(got[5 + 5 * k:10 + 5 * k]) for k in range(c["steps"])]
    return {"state": flat(v.detach() for v in state), "initial": flat(got[:5]), "controls": split, "parameters": torch.stack(got[-4:])}


def _network(c, weights, rhs):
    """Output channel 0 of the network [batch, z, y, x] for right-hand sides on its grid."""
    def split():
        at = 0
        for a, b in ((16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 64), (64, 64), (64, 32), (32, 16), (16, 16), (16, 16)):
            yield weights[at:at + 27 * a * b].reshape(27, b, a)
            at += 27 * a * b

    w = iter(split())

    def conv(x, relu=True):  # [batch, z, y, x, channels], the taps one by one
        k, (b, z, y, n, _) = next(w), x.shape
        pad = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        out = sum(pad[:, t // 9:t // 9 + z, t // 3 % 3:t // 3 % 3 + y, t % 3:t % 3 + n] @ k[t].T for t in range(27))
        return out.relu() if relu else out

    def pool(x):
        b, z, y, n, q = x.shape
        return x.reshape(b, z // 2, 2, y // 2, 2, n // 2, 2, q).mean(dim=(2, 4, 6))

    def up(x):
        for d in (1, 2, 3):
            x = x.repeat_interleave(2, dim=d)
        return x

    x = torch.zeros((*rhs.shape, 16), dtype=torch.float64, device=rhs.device)
    x[..., 0] = rhs / rhs.square().mean(dim=(1, 2, 3), keepdim=True).sqrt()
    x[..., 1] = 1.0
    e0 = conv(conv(x))
    e1 = conv(conv(pool(e0)))
    e2 = conv(conv(pool(e1)))
    m = conv(conv(pool(e2)))
    d2 = conv(up(m) + e2)
    d1 = conv(up(d2) + e1)
    d0 = conv(up(d1) + e0)
    return conv(d0, relu=False)[..., 0]


def _exact_network(c, seed):
    dev = torch.device(DEVICE if torch.cuda.is_available() else "cpu")
    rhs, p = (v.double() for v in _pairs(c, seed, dev))
    with np.load(WEIGHTS) as f:
        weights = torch.from_numpy(f["parameters"]).double().to(dev)
    if c["work"] == "predict":
        with torch.no_grad():
            return _network(c, weights, rhs).reshape(c["batch"], -1)
    weights.requires_grad_()
    grid, loss = _Grid(c, dev), 0.0
    for b in range(c["batch"]):  # the samples one by one, for memory
        g = _network(c, weights, rhs[b:b + 1])[0]
        ag, at = grid.laplacian(g), grid.laplacian(p[b])
        one = (1.0 - (g * at).sum() ** 2 / ((g * ag).sum() * (p[b] * at).sum())) / c["batch"]
        one.backward()
        loss = loss + float(one)
    return [torch.tensor([loss], dtype=torch.float64, device=dev), weights.grad]


def exact(c, seed):
    return _exact_network(c, seed) if c["work"] in ("predict", "train") else _exact_fluid(c, seed)
