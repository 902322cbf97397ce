"""Red-black sweeps with the grid in the SMs (csrc/rbgs_resident.cuh) against
the FP32 oracle's sweeps, bit for bit without a periodic axis (the oracle adds
and divides in the kernels' order, in FP32, without contraction): rows that end inside a group of 8, single rows and
planes, bricks cut short at the grid's end, one to eight groups per thread,
fixed values on every face, solid cells, an anchor cell."""
import ctypes as C

import numpy as np
import pytest

from diff_solver_b200.data import Configuration, ScalarBoundaryMode

from oracle import binding as ob

pytestmark = pytest.mark.gpu

Z, F, P = ScalarBoundaryMode.zero_gradient, ScalarBoundaryMode.fixed_value, ScalarBoundaryMode.periodic
PLUME = (Z, Z, Z, F, Z, Z)

CASES = [
    ((1, 1, 1), (F,) * 6, 3), ((1, 5, 3), (F, Z, Z, Z, Z, F), 5), ((7, 1, 4), (Z, F, F, Z, Z, Z), 5), ((8, 6, 1), PLUME, 6),
    ((9, 7, 5), (F, F, F, F, F, F), 11), ((16, 12, 10), (Z,) * 6, 9), ((23, 18, 17), (Z, F, Z, F, F, Z), 12), ((64, 40, 36), PLUME, 8),
    ((90, 61, 77), PLUME, 6), ((128, 96, 90), (F, Z, Z, F, Z, Z), 4), ((128, 130, 128), PLUME, 3), ((128, 192, 128), PLUME, 3),
    ((160, 160, 160), PLUME, 2),
    ((12, 10, 8), (P, P, Z, F, Z, Z), 6),  # a periodic axis: the general kernel
]


@pytest.mark.parametrize("res,modes,sweeps", CASES, ids=["x".join(map(str, r)) for r, _, _ in CASES])
@pytest.mark.parametrize("solid", [False, True], ids=["open", "solid"])
def test_sweeps_match_the_oracle(cuda, res, modes, sweeps, solid):
    import torch
    from diff_solver_b200 import _native as N
    from diff_solver_b200.data import Collider, Ellipsoid, Vector3
    from diff_solver_b200.model import ExecutionMode, Model
    nx, ny, nz = res
    if solid and min(res) < 5:
        pytest.skip("no room for a solid")
    cfg = Configuration(resolution=list(res), cell_size=1.0 / nx, time_step=0.5 / nx)
    for k, (face, m) in enumerate(zip(cfg.pressure_boundary.faces(), modes)):
        face.mode = m
        face.value = 0.3 * (k + 1) if m == F else 0.0
    if solid:
        cfg.colliders = [Collider(Ellipsoid(Vector3(0.45, 0.5 * ny / nx, 0.45 * nz / nx), Vector3(0.2, 0.2 * ny / nx, 0.25 * nz / nx)))]
    ctx = Model(cfg).allocate_context(ExecutionMode.forward)
    prob = ob.Problem(cfg, "f32", solver="rbgs", iterations=sweeps)
    rhs = np.random.default_rng(2).normal(size=nx * ny * nz).astype(np.float32)
    mask = ctx.domain.cell_mask if solid else None
    if solid:
        rhs[mask.cpu().numpy() != 0] = 0.0
    if ctx.domain.pressure_anchor < rhs.size:
        rhs[ctx.domain.pressure_anchor] = 0.0
    L = N.lib()
    ws = torch.full((L.xs_projection_workspace_bytes(ctx.native.grid),), 0x7F, dtype=torch.uint8, device="cuda")  # stale scratch
    b = torch.as_tensor(rhs, device="cuda")
    p = torch.full_like(b, float("nan"))
    solve = N.XsPressureSolve(N.XS_SOLVER_RED_BLACK_GAUSS_SEIDEL, sweeps, 0.0, None)
    for _ in range(2):  # and a second solve in the same scratch
        N.check("solve", L.xs_pressure_solve(None, ctx.native.grid, solve, ctx.domain.pressure_anchor, None if mask is None else mask.data_ptr(),
                                             ctx.native.pressure_boundary, b.data_ptr(), p.data_ptr(), ws.data_ptr()))
    stats = N.XsSolveStats()
    N.check("stats", L.xs_read_solve_stats(None, ws.data_ptr(), C.byref(stats)))
    assert stats.status == 0 and stats.iterations == sweeps
    want = prob.rbgs(rhs, sweeps)
    got = p.cpu().numpy()
    # the same sums in the same order; an update rounds seven times, relative to
    # values a few times the largest right-hand side or boundary value
    if P not in modes:
        assert np.array_equal(got, want)
    assert np.abs(got - want).max() <= 7 * sweeps * 2.0 ** -24 * 4 * max(np.abs(want).max(), np.abs(rhs).max())
