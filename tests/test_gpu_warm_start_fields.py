"""xs_smoke_warm_start_fields: the ring's Galerkin start of the last forward
solve and its residual, whatever the solve itself started from (the ring's
start, sweeps and coarse-grid rounds on it, the network's step, the direct
solve of the grid's operator)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS, HISTORY = 6, 3


def apply_plume(v, shape):
    """A v of the plume's pressure boundary: fixed at the top (y max), zero
    gradient elsewhere."""
    nx, ny, nz = shape
    f = np.asarray(v, np.float64).reshape(nz, ny, nx)
    out = np.zeros_like(f)
    for axis in range(3):
        d = np.diff(f, axis=axis)
        lower, upper = [slice(None)] * 3, [slice(None)] * 3
        lower[axis], upper[axis] = slice(None, -1), slice(1, None)
        out[tuple(lower)] -= d
        out[tuple(upper)] += d
    out[:, -1, :] += f[:, -1, :]
    return out.reshape(-1)


# (extents, coarsening, rounds, network)
CASES = [((32, 24, 16), 0, 0, False), ((32, 24, 16), 2, 0, False), ((33, 27, 21), 3, 0, False), ((32, 24, 16), 2, 1, False),
         ((32, 24, 16), 2, 2, False), ((32, 24, 16), 2, 3, False), ((128, 64, 32), 0, 0, True), ((128, 64, 32), 2, 0, True),
         ((128, 64, 32), 2, 2, True), ((136, 128, 72), 2, 0, False)]


@pytest.mark.parametrize("shape,coarsening,rounds,learned", CASES)
def test_fields_are_the_ring_start(cuda, shape, coarsening, rounds, learned):
    import torch
    from diff_solver_b200.data import plume_configuration
    from diff_solver_b200.model import ExecutionMode, Model, fill_parameters
    from diff_solver_b200.warm_start import WarmStartNetwork
    cfg = plume_configuration(shape)
    cfg.pressure_tolerance = 1e-7
    cfg.warm_start_history, cfg.warm_start_coarsening, cfg.warm_start_rounds = HISTORY, coarsening, rounds
    m = Model(cfg)
    ctx = m.allocate_context(ExecutionMode.forward)
    ctx.workspace.fill_(0x7F)  # stale scratch must not matter
    ctx.reset_warm_start()
    net = WarmStartNetwork(shape, factor=1, seed=4) if learned else None
    if learned:
        ctx.set_learned_warm_start(net)
    s, n = m.allocate_state(ctx), m.allocate_state(ctx)
    c, k = m.allocate_control(ctx), m.allocate_step_cache(ctx)
    q = fill_parameters(m.allocate_parameters(ctx), 0.0, -0.1, 0.5)
    g = torch.Generator().manual_seed(3)
    for t in s.velocity.components():
        t.copy_((torch.rand(t.shape, generator=g) * 0.4 - 0.2).cuda())
    previous = []
    for step in range(STEPS):
        m.forward_step(s, c, q, n, k, ctx)
        s, n = n, s
        p, b = (t.double().cpu().numpy() for t in ctx.pressure_fields())
        x0, r0 = (t.double().cpu().numpy() for t in ctx.warm_start_fields())
        a = lambda v: apply_plume(v, shape)
        # the residual is that of x0: FP32 products, an operator of norm 12
        assert np.linalg.norm(b - a(x0) - r0) <= 12 * 4 * 2.0 ** -24 * np.linalg.norm(x0) + 1e-6 * np.linalg.norm(b)
        if not previous:
            assert np.all(x0 == 0.0)
        else:
            v = np.stack(previous[-HISTORY:], axis=1)
            # in the span of the previous solutions
            w, _, rank, _ = np.linalg.lstsq(v / np.linalg.norm(v, axis=0), x0, rcond=None)
            assert np.linalg.norm(x0 - (v / np.linalg.norm(v, axis=0)) @ w) <= 1e-4 * np.linalg.norm(x0)
            # and A-norm-optimal there: its distance from the solution is the least one's
            av = np.stack([a(u) for u in v.T], axis=1)
            best = v @ np.linalg.lstsq(v.T @ av, v.T @ b, rcond=1e-12)[0]
            distance = lambda x: np.sqrt((p - x) @ a(p - x))
            assert distance(x0) <= 1.05 * distance(best) + 1e-5 * distance(0 * p), (step, distance(x0), distance(best), distance(0 * p))
            assert distance(x0) >= 0.95 * distance(best) - 1e-5 * distance(0 * p), (step, distance(x0), distance(best), distance(0 * p))
        previous.append(p)
    # a reset empties the ring, not the last solve's start
    ctx.reset_warm_start()
    again = [t.double().cpu().numpy() for t in ctx.warm_start_fields()]
    assert np.array_equal(again[0], x0) and np.array_equal(again[1], r0)
    m.forward_step(s, c, q, n, k, ctx)
    assert float(ctx.warm_start_fields()[0].abs().max()) == 0.0
    if learned:
        net.check()
