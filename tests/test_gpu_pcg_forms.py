"""The pressure solve's forms (csrc/pcg_single.cuh) at the sizes where their
index arithmetic can go wrong, against the FP64 oracle's system: rows that are
no multiple of 4, extents of one to a few cells, bricks cut short at the grid's
end, one to four groups per thread, periodic axes alone and together, solid
cells, an anchor cell, fixed values, warm starts with and without smoothing."""
import ctypes as C

import numpy as np
import pytest

from common import rel_l2
from diff_solver_b200.data import Configuration, ScalarBoundaryMode

from oracle import binding as ob

pytestmark = pytest.mark.gpu

Z, F, P = ScalarBoundaryMode.zero_gradient, ScalarBoundaryMode.fixed_value, ScalarBoundaryMode.periodic
PLUME = (Z, Z, Z, F, Z, Z)

# (extents, boundary modes, solid ball)
RESIDENT = [
    ((4, 4, 4), PLUME, False), ((1, 7, 5), PLUME, False), ((5, 1, 9), (F, Z, Z, Z, Z, Z), False), ((2, 3, 1), (P, P, Z, F, P, P), False),
    ((1, 1, 1), (F, F, F, F, F, F), False), ((7, 6, 5), (Z,) * 6, False), ((33, 17, 20), (F, Z, Z, F, F, F), True),
    ((34, 9, 31), (P, P, P, P, Z, F), True), ((35, 12, 11), (P, P, P, P, P, P), False), ((48, 40, 36), (Z,) * 6, True),
    ((64, 64, 64), PLUME, False), ((70, 61, 53), PLUME, True), ((97, 60, 59), (P, P, Z, F, P, P), True), ((90, 88, 75), PLUME, False),
]
# periodic axes of one cell, and periodic rows of 4, whose ends are one group
WRAPPED = [((4, 7, 5), (P, P, Z, F, Z, Z), False), ((8, 1, 6), (Z, F, P, P, Z, Z), False), ((12, 6, 1), (Z, F, Z, Z, P, P), False),
           ((4, 1, 9), (P, P, P, P, F, Z), False), ((4, 6, 5), (P, P, P, P, P, P), False), ((4, 128, 96), (P, P, Z, F, Z, Z), False),
           ((1200, 1, 30), (Z, Z, P, P, F, F), False), ((32, 900, 1), (F, F, Z, Z, P, P), False)]
MARCHING = [((118, 112, 101), (P, P, P, P, Z, F), True), ((121, 115, 98), PLUME, True), ((128, 112, 90), PLUME, False),
            ((700, 50, 40), PLUME, True)]


def problem(res, modes, ball, seed=3):
    cfg = Configuration(resolution=list(res), cell_size=1.0 / max(res), time_step=0.5 / max(res))
    pb = cfg.pressure_boundary
    for k, (face, m) in enumerate(zip(pb.faces(), modes)):
        face.mode = m
        face.value = 0.01 * (k + 1) if m == F and min(res) > 6 and not ball else 0.0
    prob = ob.Problem(cfg, "f64")
    nx, ny, nz = res
    z, y, x = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in (nz, ny, nx)], indexing="ij")
    mask = None
    if ball:
        mask = (((x - 0.45) ** 2 + (y - 0.5) ** 2 + (z - 0.4) ** 2) < 0.04).astype(np.uint32).ravel()
    rhs = np.random.default_rng(seed).normal(size=nx * ny * nz) + np.sin(5 * x + 2 * y - 3 * z).ravel()
    if F not in modes:  # an anchored system: a source without sum, as a closed box has
        fluid = np.ones(rhs.size, bool) if mask is None else mask == 0
        rhs[fluid] -= rhs[fluid].mean()
    return cfg, prob, mask, rhs.astype(np.float32)


class Solve:
    def __init__(self, cfg, mask, rhs, anchor):
        import torch
        from diff_solver_b200 import _native as N
        from diff_solver_b200.model import scalar_boundary
        self.N, self.L, self.torch = N, N.lib(), torch
        self.g = N.XsGrid(*[int(v) for v in cfg.resolution], float(cfg.cell_size), float(cfg.time_step))
        self.pb, self.anchor = scalar_boundary(cfg.pressure_boundary), anchor
        self.rhs = torch.as_tensor(rhs, device="cuda")
        self.mask = None if mask is None else torch.as_tensor(mask.astype(np.int32), device="cuda")
        # stale scratch must not matter
        self.ws = torch.full((self.L.xs_projection_workspace_bytes(self.g),), 0x7F, dtype=torch.uint8, device="cuda")

    def __call__(self, tolerance, guess=None, scale=0, iterations=20000):
        N = self.N
        s = N.XsPressureSolve(N.XS_SOLVER_JACOBI_PCG, iterations, tolerance, None if guess is None else guess.data_ptr())
        s.scale_guess = scale
        p = self.torch.full_like(self.rhs, float("nan"))
        N.check("solve", self.L.xs_pressure_solve(None, self.g, s, self.anchor, None if self.mask is None else self.mask.data_ptr(), self.pb,
                                                  self.rhs.data_ptr(), p.data_ptr(), self.ws.data_ptr()))
        st = N.XsSolveStats()
        N.check("stats", self.L.xs_read_solve_stats(None, self.ws.data_ptr(), C.byref(st)))
        return p, st


def anchor_of(modes, mask, n):
    if F in modes:
        return n
    return 0 if mask is None else int(np.argmax(mask == 0))


def masked_system(cfg, prob, mask, anchor, rhs):
    """A and b of the system in FP64 on the host, as functions of flat arrays."""
    nx, ny, nz = (int(v) for v in cfg.resolution)
    solid = np.zeros(nx * ny * nz, bool) if mask is None else mask.astype(bool)
    fluid = (~solid).reshape(nz, ny, nx).astype(float)
    faces = cfg.pressure_boundary.faces()

    def neighbours(v, fixed):
        total, count = np.zeros_like(v), np.zeros_like(v)
        for d in range(3):
            ax, per = 2 - d, faces[2 * d].mode == P and faces[2 * d + 1].mode == P
            for side in (0, 1):
                sh = -1 if side else 1
                nb, there = np.roll(v * fluid, sh, ax), np.roll(fluid, sh, ax)
                if not per:
                    edge = [slice(None)] * 3
                    edge[ax] = -1 if side else 0
                    f = faces[2 * d + side]
                    nb[tuple(edge)] = f.value if fixed and f.mode == F else 0.0
                    there[tuple(edge)] = 1.0 if f.mode == F else 0.0
                total, count = total + nb, count + there
        return total, count

    _, count = neighbours(fluid, False)
    active = (fluid.ravel() > 0) & (count.ravel() > 0)
    if anchor < active.size:
        active[anchor] = False

    def apply(x):
        v = np.where(active, x, 0.0).reshape(nz, ny, nx)
        total, _ = neighbours(v, False)
        return np.where(active, (count * v - total).ravel(), 0.0)

    fixed, _ = neighbours(np.zeros((nz, ny, nx)), True)
    return apply, np.where(active, rhs.astype(np.float64) + fixed.ravel(), 0.0), active


FORMS = RESIDENT + WRAPPED + MARCHING


@pytest.mark.parametrize("res,modes,ball", FORMS, ids=["x".join(map(str, r)) + ("-solid" if b else "") for r, _, b in FORMS])
def test_solutions_satisfy_the_system(cuda, res, modes, ball):
    cfg, prob, mask, rhs = problem(res, modes, ball)
    n = int(np.prod(res))
    anchor = anchor_of(modes, mask, n)
    apply, b, active = masked_system(cfg, prob, mask, anchor, rhs)
    solve = Solve(cfg, mask, rhs, anchor)
    p, st = solve(1e-8)
    x = p.cpu().numpy().astype(np.float64)
    assert st.status == 0 and st.final_residual <= 1e-8
    assert np.isfinite(x).all() and not x[~active].any()
    # the solution is stored in 32 bits: rounding it moves the residual by at
    # most the operator's norm (12) times half a unit in the last place
    bound = 1e-8 * np.linalg.norm(b) + 12 * 2.0 ** -24 * np.linalg.norm(x)
    assert np.linalg.norm(b - apply(x)) <= 1.01 * bound, (np.linalg.norm(b - apply(x)), bound)
    if mask is None and n <= 64 ** 3 and active.sum() > 1:
        want, ost = prob.pcg(b, 20000, 1e-12) if anchor >= n else (None, None)
        if want is not None and not any(f.value for f in cfg.pressure_boundary.faces()):
            # residual 1e-8, condition number below 4 max(res)^2 / 2
            assert rel_l2(x, want) <= 1e-8 * 2 * max(res) ** 2 + 2.0 ** -24
    if active.sum() < 50:
        return
    # a start near the solution converges to the same, with smoothing on the way
    torch = solve.torch
    near = (p * (1 + 1e-4 * torch.sin(0.0371 * torch.arange(n, device="cuda", dtype=torch.float32)))).contiguous()
    q, sq = solve(1e-7, guess=near)
    assert sq.status == 0 and sq.final_residual <= 1e-7 and sq.warm_start_used == 1 and sq.iterations < st.iterations
    bound = 1e-7 * np.linalg.norm(b) + 12 * 2.0 ** -24 * np.linalg.norm(x)
    assert np.linalg.norm(b - apply(q.cpu().numpy().astype(np.float64))) <= 1.01 * bound
    # the energy-optimal scale undoes a factor; a useless guess is dropped and the solve is the cold one
    _, scaled = solve(1e-6, guess=(2.5 * p).contiguous(), scale=1)
    assert abs(scaled.guess_scale - 0.4) < 1e-3 and scaled.warm_start_used == 1
    _, cold = solve(1e-6)
    _, dropped = solve(1e-6, guess=torch.full_like(p, 1e4))
    assert dropped.warm_start_used == 0 and dropped.iterations == cold.iterations and dropped.status == 0
    # the iteration cap
    _, capped = solve(1e-8, iterations=5)
    assert capped.status == 2 and capped.iterations == 5


def test_the_same_solve_twice_is_the_same(cuda):
    """Sums are taken in a fixed order: equal inputs, equal bits."""
    for res, modes, ball in (RESIDENT[11], MARCHING[1]):
        cfg, _, mask, rhs = problem(res, modes, ball)
        solve = Solve(cfg, mask, rhs, anchor_of(modes, mask, int(np.prod(res))))
        a, b = solve(1e-6)[0], solve(1e-6)[0]
        assert solve.torch.equal(a, b)
