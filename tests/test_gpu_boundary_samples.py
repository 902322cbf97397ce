"""Advection samples beyond the domain: every pair of boundary modes, axes of a
few nodes, traces of several cells and of more than one period, against the
node rules written out in FP64 (operators.cu:88-134)."""
import ctypes as C
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def nodes(v, c, size, period, per, fixed):
    """Values of v at integer coordinates c (three arrays).  fixed(d, low) gives
    the fixed value at that end of axis d, or None."""
    at = [np.mod(c[d], period[d]) if per[d] else np.clip(c[d], 0, size[d] - 1) for d in range(3)]
    out = v[at[2], at[1], at[0]].astype(np.float64)
    for d in (2, 1, 0):  # the first axis' value counts
        for low, beyond in ((False, c[d] >= size[d]), (True, c[d] < 0)):
            value = fixed(d, low)
            if value is not None:
                out = np.where(beyond, value, out)
    return out


def sample(v, p, offset, size, period, per, fixed):
    g = [p[d] - offset[d] for d in range(3)]
    c0 = [np.floor(x).astype(np.int64) for x in g]
    t = [g[d] - c0[d] for d in range(3)]
    out = 0.0
    for e in itertools.product((0, 1), repeat=3):
        w = 1.0
        for d in range(3):
            w = w * (t[d] if e[d] else 1.0 - t[d])
        out = out + w * nodes(v, [c0[d] + e[d] for d in range(3)], size, period, per, fixed)
    return out


@pytest.mark.parametrize("h", [0.03, 1.0 / 32.0])
@pytest.mark.parametrize("res", [(5, 4, 3), (35, 6, 5), (3, 9, 17)])
@pytest.mark.parametrize("modes", [(0, 0), (1, 1), (2, 2), (3, 3), (0, 1), (1, 0), (2, 0), (1, 2)])
def test_samples_beyond_the_domain(cuda, modes, res, h):
    """Fixed, free, normal-fixed and periodic ends (scalars: fixed, free,
    periodic).  Positions are FP32 in the kernels, a few 1e-7 of a cell's
    coordinate off, and the samples' slopes are below 2 per cell and axis: 1e-4
    of an error leaves a factor of ten."""
    import torch
    from diff_solver_b200 import _native as N
    L = N.lib()
    rng = np.random.default_rng(res[0] + 10 * modes[0] + modes[1])
    n = res
    dt = 0.02
    g = N.XsGrid(n[0], n[1], n[2], h, dt)
    vb = N.XsVelocityBoundary()
    sb = N.XsScalarBoundary()
    smode = {0: 0, 1: 1, 2: 1, 3: 2}
    for f in range(6):
        vb.modes[f] = modes[f & 1]
        sb.modes[f] = smode[modes[f & 1]]
        sb.values[f] = float(np.float32(rng.uniform(-1, 1)))
        for a in range(3):
            vb.values[3 * f + a] = float(np.float32(rng.uniform(-1, 1)))
    per = [modes == (3, 3)] * 3
    size = [[n[d] + (d == a) for d in range(3)] for a in range(3)]
    # smooth in space, up to 2.5 cells a step
    u = [(2.5 * h / dt * rng.uniform(-1, 1, (size[a][2], size[a][1], size[a][0]))).astype(np.float32) for a in range(3)]
    for a in range(3):
        for f in range(6):
            vb.values[3 * f + a] *= 0.5 * h / dt
    s = rng.uniform(-1, 1, (n[2], n[1], n[0])).astype(np.float32)

    def face_fixed(a):
        def fixed(d, low):
            f = 2 * d + (0 if low else 1)
            return vb.values[3 * f + a] if vb.modes[f] == 0 or (vb.modes[f] == 2 and a == d) else None
        return fixed

    def scalar_fixed(d, low):
        f = 2 * d + (0 if low else 1)
        if sb.modes[f] == 0:
            return sb.values[f]
        # (a coordinate below 0 also counts as beyond the upper end)
        return sb.values[2 * d + 1] if low and sb.modes[2 * d + 1] == 0 else None

    def velocity(p):
        return [sample(u[a], p, [0.0 if d == a else 0.5 for d in range(3)], size[a], n, per, face_fixed(a)) for a in range(3)]

    def trace(p):
        v0 = velocity(p)
        v1 = velocity([p[d] - 0.5 * dt / h * v0[d] for d in range(3)])
        end = [p[d] - dt / h * v1[d] for d in range(3)]
        return [end[d] if per[d] else np.clip(end[d], 0.0, n[d]) for d in range(3)]

    def positions(shape, offset):
        z, y, x = np.meshgrid(*(np.arange(shape[d], dtype=np.float64) for d in (2, 1, 0)), indexing="ij")
        return [x + offset[0], y + offset[1], z + offset[2]]

    dev = torch.device("cuda")
    ud = [torch.as_tensor(a, device=dev) for a in u]
    out = [torch.zeros_like(a) for a in ud]
    sd, so = torch.as_tensor(s, device=dev), torch.zeros(s.shape, dtype=torch.float32, device=dev)
    N.check("advect", L.xs_advect_velocity_forward(None, g, None, N.vec(ud), vb, N.vec(out)))
    N.check("scalar", L.xs_advect_scalar_forward(None, g, None, None, C.c_void_p(sd.data_ptr()), N.vec(ud), sb, vb, C.c_void_p(so.data_ptr())))
    torch.cuda.synchronize()
    for a in range(3):
        off = [0.0 if d == a else 0.5 for d in range(3)]
        want = sample(u[a], trace(positions(size[a], off)), off, size[a], n, per, face_fixed(a))
        scale = 2.5 * h / dt
        assert np.abs(out[a].cpu().numpy() - want).max() < 1e-4 * scale, (modes, res, a)
    want = sample(s, trace(positions(n, [0.5] * 3)), [0.5] * 3, list(n), n, per, scalar_fixed)
    assert np.abs(so.cpu().numpy() - want).max() < 1e-4, (modes, res)
