"""The direct solve that starts warm-started pressure solves (csrc/direct.cu)
over the axes, ends and extents its index arithmetic and formulas distinguish:
even, odd and short extents, extents past a tile of 64 modes and a segment of
32 values, equal ends of each kind, periodic axes, unequal ends on the
tridiagonal axis, y or z tridiagonal, aligned and ragged rows."""
import numpy as np
import pytest

from common import rel_l2, seeded_control, seeded_state
from diff_solver_b200.data import Configuration, ScalarBoundaryMode, VelocityBoundaryMode

pytestmark = pytest.mark.gpu

Z, F, P = ScalarBoundaryMode.zero_gradient, ScalarBoundaryMode.fixed_value, ScalarBoundaryMode.periodic

# (extents, coarsening, pressure boundary)
CASES = [
    ((16, 24, 32), 2, (Z, Z, Z, F, Z, Z)),
    ((33, 27, 21), 3, (Z, Z, F, Z, Z, Z)),
    ((9, 6, 15), 3, (F, F, F, F, F, F)),
    ((4, 4, 4), 2, (Z, Z, Z, F, Z, Z)),
    ((45, 66, 39), 3, (P, P, Z, F, P, P)),
    ((130, 34, 70), 2, (P, P, F, F, Z, Z)),
    ((35, 65, 25), 5, (F, F, Z, Z, P, P)),
    ((40, 36, 34), 2, (Z, Z, P, P, Z, F)),    # z tridiagonal: y is periodic
    ((36, 33, 63), 3, (P, P, Z, Z, F, Z)),    # ... z has unequal ends
    ((4, 48, 40), 2, (P, P, Z, F, Z, Z)),     # a periodic row of one group
    ((4, 160, 120), 2, (P, P, Z, F, Z, Z)),
    ((136, 128, 72), 2, (Z, Z, Z, F, Z, Z)),  # two parts: past 1.2 M cells
    ((111, 108, 105), 3, (P, P, F, Z, F, F)),
    ((264, 80, 60), 2, (Z, Z, Z, F, Z, Z)),   # an axis of more than 256 cells
]


def configuration(res, coarsening, modes, warm):
    cfg = Configuration(resolution=list(res), cell_size=1.0 / res[0], time_step=0.5 / res[0], vorticity_confinement_enabled=False)
    for face, vface, m in zip(cfg.pressure_boundary.faces(), cfg.velocity_boundary.faces(), modes):
        face.mode = m
        vface.mode = {Z: VelocityBoundaryMode.normal_fixed_tangent_zero_gradient, F: VelocityBoundaryMode.zero_gradient,
                      P: VelocityBoundaryMode.periodic}[m]
    for b in (cfg.density_boundary, cfg.temperature_boundary):
        for face, m in zip(b.faces(), modes):
            face.mode = P if m == P else Z
    cfg.pressure_max_iterations = 20000
    if warm:
        cfg.warm_start_history, cfg.warm_start_coarsening = 2, coarsening
    return cfg


def context(cfg, seed):
    from common import to_model_control, to_model_state
    from diff_solver_b200.model import ExecutionMode, Model, fill_parameters
    m = Model(cfg)
    ctx = m.allocate_context(ExecutionMode.differentiable)
    ctx.workspace.fill_(0x7F)  # stale scratch must not matter
    ctx.reset_warm_start()
    res = tuple(cfg.resolution)
    return (m, ctx, to_model_state(m, ctx, seeded_state(res, seed=seed, amp=0.1)), to_model_control(m, ctx, seeded_control(res, seed=seed + 1)),
            fill_parameters(m.allocate_parameters(ctx), 0.0, -0.1, 0.5))


def relative_residual(p, b, res, modes):
    """|b - A p| / |b| in FP64 (fixed values are 0 in these cases)."""
    f = np.asarray(p, np.float64).reshape(res[::-1])
    out = np.zeros_like(f)
    for d in range(3):
        axis = 2 - d
        g = np.moveaxis(f, axis, 0)
        o = np.moveaxis(out, axis, 0)
        o[:-1] += g[:-1] - g[1:]
        o[1:] += g[1:] - g[:-1]
        if modes[2 * d] == P:
            o[0] += g[0] - g[-1]
            o[-1] += g[-1] - g[0]
        else:
            o[0] += g[0] if modes[2 * d] == F else 0.0
            o[-1] += g[-1] if modes[2 * d + 1] == F else 0.0
    return float(np.linalg.norm(b - out.reshape(-1)) / np.linalg.norm(b))


@pytest.mark.parametrize("res,coarsening,modes", CASES, ids=["x".join(map(str, r)) for r, _, _ in CASES])
def test_start_solves_the_system(cuda, res, coarsening, modes):
    from diff_solver_b200.model import tensors_of
    out, n = {}, int(np.prod(res))
    for warm in (False, True):
        m, ctx, state, control, par = context(configuration(res, coarsening, modes, warm), 7)
        nxt, cache = m.allocate_state(ctx), m.allocate_step_cache(ctx)
        m.forward_step(state, control, par, nxt, cache, ctx)
        forward = ctx.read_solve_stats()
        pressure, rhs = (t.double().cpu().numpy() for t in ctx.pressure_fields())
        seed, prev = m.allocate_state_adjoint(ctx), m.allocate_state_adjoint(ctx)
        for t, s in zip(seed.velocity.components(), state.velocity.components()):
            t.copy_(s)
        m.vjp_step(state, control, par, nxt, cache, seed, prev, m.allocate_control_adjoint(ctx), m.allocate_parameter_adjoint(ctx), ctx)
        adjoint = ctx.read_solve_stats()
        out[warm] = ([t.cpu().numpy() for t in tensors_of(nxt)], [t.cpu().numpy() for t in prev.velocity.components()], forward, adjoint)
    # one part: FP32 transforms and tridiagonal sweeps, some tens of roundings of
    # x, moved by an operator of norm 12; of the adjoint's x only the most its
    # norm can be is known here, (2 max(res) / pi)^2 times that of its right-hand
    # side, and that states like these stay far from it (1.4e-5 measured).  Two
    # parts: the second takes the first's residual down as far again
    # (2e-12 measured), further than any one FP32 vector can (the FP32 rounding
    # of the solution: 4e-8)
    roundings = 12 * 32 * 2.0 ** -24
    twice = n >= 1200000
    bounds = [1e-9, 1e-9] if twice else [roundings * np.linalg.norm(pressure) / np.linalg.norm(rhs),
                                         min(roundings * (2 * max(res) / np.pi) ** 2, 1e-4)]
    if twice:
        assert relative_residual(pressure, rhs, res, modes) > 1e-8
        assert all(s["iterations"] == 0 for s in out[True][2:])
    for stats, bound in zip(out[True][2:], bounds):
        assert stats["status"] == 0 and stats["warm_start_used"] == 1 and stats["coarse_iterations"] == 0
        assert stats["initial_residual"] <= bound, (stats["initial_residual"], bound)
        assert stats["final_residual"] <= 1e-6
    for warm, plain in zip(out[True][2:], out[False][2:]):
        assert warm["iterations"] <= max(3, plain["iterations"] // 2)
    # both within the solver's tolerance of the same step and the same adjoint
    for a, b in zip(out[True][0] + out[True][1], out[False][0] + out[False][1]):
        if np.linalg.norm(b) > 0:
            assert rel_l2(a, b) < 1e-4, rel_l2(a, b)


def test_the_network_works_on_the_residual_of_the_start(cuda):
    """The residual an almost exact start leaves is formed in FP64 before the
    network's step: with an FP32 A x most of it is that product's rounding.
    The trained network at factor 1 then leaves 0.14 of the start's residual
    (0.24 with FP32 products)."""
    import os
    import torch
    from common import ROOT
    from diff_solver_b200.data import plume_configuration
    from diff_solver_b200.model import ExecutionMode, Model, fill_parameters
    from diff_solver_b200.warm_start import WarmStartNetwork
    res = (128, 64, 32)
    cfg = plume_configuration(res)
    cfg.warm_start_history, cfg.warm_start_coarsening = 5, 2
    net = WarmStartNetwork(res, factor=1)
    net.load(os.path.join(ROOT, "diff_solver_b200", "weights", "warm_start_128.npz"))
    left = []
    for network in (None, net):
        m = Model(cfg)
        ctx = m.allocate_context(ExecutionMode.forward)
        if network is not None:
            ctx.set_learned_warm_start(network)
        s, n = m.allocate_state(ctx), m.allocate_state(ctx)
        c, k = m.allocate_control(ctx), m.allocate_step_cache(ctx)
        q = fill_parameters(m.allocate_parameters(ctx), 0.0, -0.1, 0.5)
        g = torch.Generator().manual_seed(0)
        for t in s.velocity.components():
            t.copy_((torch.rand(t.shape, generator=g) * 0.02 - 0.01).cuda())
        initial = []
        for _ in range(30):
            m.forward_step(s, c, q, n, k, ctx)
            s, n = n, s
            initial.append(ctx.read_solve_stats()["initial_residual"])
        left.append(np.mean(initial[10:]))
    net.check()
    print(left)
    assert left[1] < 0.18 * left[0], left


def test_settings_keep_the_rounds(cuda):
    """A number of rounds set by the caller, and grids that do not separate,
    keep the ring and the rounds."""
    import copy
    modes = (Z, Z, Z, F, Z, Z)
    base = configuration((32, 32, 32), 2, modes, True)
    rounds = copy.deepcopy(base)
    rounds.warm_start_rounds = 1
    two = configuration((32, 32, 32), 2, (Z, F, Z, F, Z, Z), True)  # two axes with unequal ends
    closed = configuration((32, 32, 32), 2, (Z,) * 6, True)
    closed.pressure_boundary.y_max.mode = Z
    starts = []
    for cfg in (base, rounds, two, closed):
        m, ctx, state, control, par = context(cfg, 3)
        nxt, cache = m.allocate_state(ctx), m.allocate_step_cache(ctx)
        for _ in range(4):
            m.forward_step(state, control, par, nxt, cache, ctx)
            state, nxt = nxt, state
        st = ctx.read_solve_stats()
        assert st["status"] == 0 and st["final_residual"] <= 1e-6
        starts.append(st["initial_residual"])
    print(starts)
    assert starts[0] < 1e-4 and all(s > 2 * starts[0] for s in starts[1:]), starts
