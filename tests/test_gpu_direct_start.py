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


@pytest.mark.parametrize("res,coarsening,modes", CASES, ids=["x".join(map(str, r)) for r, _, _ in CASES])
def test_start_solves_the_system(cuda, res, coarsening, modes):
    from diff_solver_b200.model import tensors_of
    out, n = {}, int(np.prod(res))
    for warm in (False, True):
        m, ctx, state, control, par = context(configuration(res, coarsening, modes, warm), 7)
        nxt, cache = m.allocate_state(ctx), m.allocate_step_cache(ctx)
        m.forward_step(state, control, par, nxt, cache, ctx)
        forward = ctx.read_solve_stats()
        seed, prev = m.allocate_state_adjoint(ctx), m.allocate_state_adjoint(ctx)
        for t, s in zip(seed.velocity.components(), state.velocity.components()):
            t.copy_(s)
        m.vjp_step(state, control, par, nxt, cache, seed, prev, m.allocate_control_adjoint(ctx), m.allocate_parameter_adjoint(ctx), ctx)
        adjoint = ctx.read_solve_stats()
        out[warm] = ([t.cpu().numpy() for t in tensors_of(nxt)], [t.cpu().numpy() for t in prev.velocity.components()], forward, adjoint)
    # FP32 transforms and tridiagonal sweeps: some tens of roundings of x, whose
    # norm is at most (2 max(res) / pi)^2 times b's, moved by an operator of norm 12
    part = 12 * 32 * 2.0 ** -24 * (2 * max(res) / np.pi) ** 2
    bound = min(part, 0.05) ** (2 if n >= 1200000 else 1)
    for stats in out[True][2:]:
        assert stats["status"] == 0 and stats["warm_start_used"] == 1 and stats["coarse_iterations"] == 0
        assert stats["initial_residual"] <= bound, (stats["initial_residual"], bound)
        assert stats["final_residual"] <= 1e-6
    for warm, plain in zip(out[True][2:], out[False][2:]):
        assert warm["iterations"] <= max(3, plain["iterations"] // 2)
    # both within the solver's tolerance of the same step and the same adjoint
    for a, b in zip(out[True][0] + out[True][1], out[False][0] + out[False][1]):
        if np.linalg.norm(b) > 0:
            assert rel_l2(a, b) < 1e-4, rel_l2(a, b)


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
