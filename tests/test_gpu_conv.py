"""tcgen05 3x3x3 convolutions against a plain PyTorch FP32 reference of the
same operation (BF16-rounded operands)."""
import itertools

import pytest

pytestmark = pytest.mark.gpu


def reference_conv(x, w, bias, relu):
    """x: [B, Z, Y, X, Cin] float; w: [27, Cout, Cin]; NDHWC out."""
    import torch
    cin, cout = x.shape[-1], w.shape[1]
    wt = w.reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2).contiguous()  # [co, ci, dz, dy, dx]
    y = torch.nn.functional.conv3d(x.permute(0, 4, 1, 2, 3), wt, bias=bias, padding=1)
    y = y.permute(0, 2, 3, 4, 1)
    return torch.relu(y) if relu else y


@pytest.mark.parametrize("cin,cout,shape", [(c, d, s) for (c, d), s in itertools.product(
    [(16, 16), (16, 32), (32, 64), (64, 64), (64, 16), (32, 32)], [(16, 16, 6), (128, 2, 3), (8, 8, 6), (4, 8, 8)])])
def test_conv_matches_torch(cuda, cin, cout, shape):
    import torch
    from diff_solver_b200 import _native as N
    nx, ny, nz = shape
    batch = 2
    g = torch.Generator(device="cpu").manual_seed(cin * 100 + cout)
    x = torch.randn(batch, nz, ny, nx, cin, generator=g).to(torch.bfloat16)
    w = (torch.randn(27, cout, cin, generator=g) / (27 * cin) ** 0.5).to(torch.bfloat16)
    bias = torch.randn(cout, generator=g).float()
    xd, wd, bd = x.cuda(), w.cuda(), bias.cuda()
    out = torch.zeros(batch, nz, ny, nx, cout, dtype=torch.bfloat16, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for relu in (0, 1):
        N.check("conv", N.lib().xs_conv3d_bf16(None, batch, nx, ny, nz, cin, cout, xd.data_ptr(), wd.data_ptr(), bd.data_ptr(),
                                               out.data_ptr(), relu, err.data_ptr()))
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        want = reference_conv(x.float(), w.float(), bias, relu)
        got = out.float().cpu()
        rel = (got - want).norm() / want.norm()
        assert rel < 1e-2, (cin, cout, shape, relu, float(rel))


@pytest.mark.parametrize("cin,cout,shape,batch", [
    (16, 16, (16, 16, 6), 2), (16, 32, (128, 2, 3), 1), (32, 64, (16, 16, 4), 2), (64, 64, (32, 8, 5), 1),
    (64, 16, (16, 8, 7), 2), (32, 32, (64, 4, 3), 3), (64, 32, (16, 16, 16), 1),
    # volumes whose x-y planes hold fewer than 128 voxels: tiles span several z planes
    (16, 16, (8, 8, 6), 2), (32, 64, (4, 8, 8), 1), (64, 64, (8, 8, 4), 2)])
def test_conv_gradients_match_torch(cuda, cin, cout, shape, batch):
    """Weight gradient (tcgen05, MN-major operands) and input gradient (the
    forward kernel with flipped, transposed weights) against autograd."""
    import torch
    from diff_solver_b200 import _native as N
    L = N.lib()
    nx, ny, nz = shape
    g = torch.Generator(device="cpu").manual_seed(7 * cin + cout + nz)
    x = torch.randn(batch, nz, ny, nx, cin, generator=g).to(torch.bfloat16)
    w = (torch.randn(27, cout, cin, generator=g) / (27 * cin) ** 0.5).to(torch.bfloat16)
    dy = torch.randn(batch, nz, ny, nx, cout, generator=g).to(torch.bfloat16)

    xf = x.float().requires_grad_(True)
    wf = w.float().requires_grad_(True)
    y = reference_conv(xf, wf, None, False)
    y.backward(dy.float())

    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.empty(L.xs_conv3d_weight_grad_scratch_floats(batch, nx, ny, nz, cin, cout), dtype=torch.float32, device="cuda")
    dw = torch.full((27, cout, cin), 3.0, dtype=torch.float32, device="cuda")
    xd, dyd = x.cuda(), dy.cuda()
    for accumulate in (0, 1):
        N.check("wgrad", L.xs_conv3d_weight_grad_bf16(None, batch, nx, ny, nz, cin, cout, xd.data_ptr(), dyd.data_ptr(),
                                                       scratch.data_ptr(), dw.data_ptr(), accumulate, err.data_ptr()))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    got = dw.cpu() / 2.0  # accumulated twice
    rel = (got - wf.grad).norm() / wf.grad.norm()
    assert rel < 1e-4, (cin, cout, shape, float(rel))

    # input gradient: conv(dY, W') with W'[t][ci][co] = W[26 - t][co][ci]
    wt = w.flip(0).transpose(1, 2).contiguous().cuda()
    dx = torch.zeros(batch, nz, ny, nx, cin, dtype=torch.bfloat16, device="cuda")
    N.check("dgrad", L.xs_conv3d_bf16(None, batch, nx, ny, nz, cout, cin, dyd.data_ptr(), wt.data_ptr(), None, dx.data_ptr(), 0,
                                      err.data_ptr()))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    rel = (dx.float().cpu() - xf.grad).norm() / xf.grad.norm()
    assert rel < 1e-2, (cin, cout, shape, float(rel))


@pytest.mark.parametrize("cout,shape,batch", [
    (16, (64, 48, 40), 1), (16, (16, 16, 98), 4), (16, (8, 48, 75), 4), (16, (32, 33 * 4, 26), 1),
    (32, (128, 37, 22), 1), (32, (32, 32, 25), 4), (64, (64, 26, 61), 1), (64, (256, 21, 19), 1)])
def test_conv_from_halo_slabs(cuda, cout, shape, batch):
    """Volumes of 100,000 voxels and more with 16 input channels: ragged strips
    of rows and layers of planes, several tiles per plane and per TMEM lane
    block, rows longer than a tile.  Against PyTorch FP32, and, where the
    samples by themselves take the kernel of shifted boxes, against that: the
    two differ by the order of FP32 sums of 432 products below 1 in
    magnitude, so by one BF16 step where a sum lies beside a rounding edge."""
    import torch
    from diff_solver_b200 import _native as N
    cin = 16
    nx, ny, nz = shape
    assert nx * ny * nz * batch >= 100000
    g = torch.Generator(device="cpu").manual_seed(cout + nx)
    x = torch.randn(batch, nz, ny, nx, cin, generator=g).to(torch.bfloat16)
    w = (torch.randn(27, cout, cin, generator=g) / (27 * cin) ** 0.5).to(torch.bfloat16)
    bias = torch.randn(cout, generator=g).float()
    xd, wd, bd = x.cuda(), w.cuda(), bias.cuda()
    out = torch.full((batch, nz, ny, nx, cout), 7.0, dtype=torch.bfloat16, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def conv(samples, src, dst, relu):
        N.check("conv", N.lib().xs_conv3d_bf16(None, samples, nx, ny, nz, cin, cout, src.data_ptr(), wd.data_ptr(), bd.data_ptr(), dst.data_ptr(),
                                               relu, err.data_ptr()))

    for relu in (0, 1):
        conv(batch, xd, out, relu)
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        want = reference_conv(x.float(), w.float(), bias, relu)
        got = out.float().cpu()
        assert (got - want).norm() / want.norm() < 1e-2
        # each sum is within BF16 rounding (2^-9) and FP32 accumulation of the reference
        assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all())
    if batch > 1:
        one = torch.empty_like(out)
        for b in range(batch):
            conv(1, xd[b], one[b], 1)
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        assert bool(((one.float() - out.float()).abs() <= 2.0 ** -7 * one.float().abs() + 1e-4).all())


@pytest.mark.parametrize("cin,cout,shape,batch", [(32, 16, (32, 32, 37), 1), (32, 32, (32, 32, 38), 1), (32, 64, (64, 64, 19), 1), (16, 64, (32, 32, 74), 1),
                                                  (64, 16, (32, 64, 38), 1), (64, 32, (64, 36, 33), 1), (64, 64, (128, 37, 17), 1), (32, 16, (64, 64, 33), 2)])
def test_conv_on_either_side_of_the_deep_stages(cuda, cin, cout, shape, batch):
    """Numbers of 128-voxel tiles at, just past and well past those that take
    deep stages (296 and 592), as many CTAs as an SM holds and more."""
    import torch
    from diff_solver_b200 import _native as N
    nx, ny, nz = shape
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn(batch, nz, ny, nx, cin, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(27, cout, cin, generator=g, device="cuda") / (27 * cin) ** 0.5).to(torch.bfloat16)
    out = torch.full((batch, nz, ny, nx, cout), float("nan"), dtype=torch.bfloat16, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    N.check("conv", N.lib().xs_conv3d_bf16(None, batch, nx, ny, nz, cin, cout, x.data_ptr(), w.data_ptr(), None, out.data_ptr(), 0, err.data_ptr()))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    want = reference_conv(x.double(), w.double(), None, False)
    # exact products, FP32 sums of 27 cin of them, one rounding to BF16
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 27 * cin * 2.0 ** -24).all())


@pytest.mark.parametrize("cin,cout,shape,batch", [(16, 16, (32, 32, 32), 1), (16, 32, (64, 30, 18), 1), (32, 32, (16, 24, 50), 2),
                                                  (16, 16, (8, 16, 30), 8), (16, 16, (16, 16, 8), 2)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")], ids=["inf", "nan"])
def test_conv_weight_gradient_of_values_that_are_not_finite(cuda, cin, cout, shape, batch, value):
    """A voxel of the input that is infinite or NaN reaches the taps that pair
    it with an output gradient, and no other: voxels in the corners, on the
    faces and inside, from slabs and (the last shape) from boxes."""
    import torch
    from diff_solver_b200 import _native as N
    L = N.lib()
    nx, ny, nz = shape
    g = torch.Generator(device="cpu").manual_seed(11)
    clean = torch.randn(batch, nz, ny, nx, cin, generator=g).to(torch.bfloat16).cuda()
    dy = torch.randn(batch, nz, ny, nx, cout, generator=g).to(torch.bfloat16).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.full((L.xs_conv3d_weight_grad_scratch_floats(batch, nx, ny, nz, cin, cout),), float("nan"), device="cuda")
    for z, y, x in ((0, 0, 0), (nz - 1, ny - 1, nx - 1), (nz // 2, ny // 2, nx - 1), (nz // 2, 0, nx // 2), (0, ny // 2, nx // 2),
                    (nz - 1, ny // 3, 0), (nz // 2, ny // 2, nx // 2), (nz // 2, ny // 2, 0)):
        xd = clean.clone()
        xd[batch - 1, z, y, x, 5] = value
        padded = torch.nn.functional.pad(xd.double(), (0, 0, 1, 1, 1, 1, 1, 1))
        want = torch.stack([torch.einsum("bzyxi,bzyxo->oi", padded[:, dz:dz + nz, ddy:ddy + ny, dx:dx + nx], dy.double())
                            for dz, ddy, dx in itertools.product(range(3), repeat=3)])
        dw = torch.zeros((27, cout, cin), dtype=torch.float32, device="cuda")
        N.check("wgrad", L.xs_conv3d_weight_grad_bf16(None, batch, nx, ny, nz, cin, cout, xd.data_ptr(), dy.data_ptr(), scratch.data_ptr(),
                                                      dw.data_ptr(), 0, err.data_ptr()))
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        finite = torch.isfinite(want)
        assert torch.equal(torch.isfinite(dw), finite), (z, y, x)
        assert torch.equal(torch.isnan(dw), torch.isnan(want)) and torch.equal(dw[torch.isinf(want)].double(), want[torch.isinf(want)])
        # (FP64 sums of the same products: as in the test below)
        assert float((dw.double() - want)[finite].norm() / want[finite].norm()) < 1e-5


@pytest.mark.parametrize("cin,cout,shape,batch", [
    (16, 16, (64, 48, 40), 1), (16, 16, (16, 24, 131), 2), (16, 32, (32, 36, 30), 3), (32, 16, (64, 26, 31), 2), (32, 32, (128, 37, 22), 1),
    (16, 16, (4, 64, 100), 4), (32, 32, (8, 48, 140), 2), (16, 16, (256, 21, 19), 1), (16, 16, (128, 800, 1), 1),
    (16, 16, (16, 24, 79), 1), (32, 32, (2, 128, 120), 1)])
def test_conv_weight_gradient_from_slabs(cuda, cin, cout, shape, batch):
    """Volumes of 30,000 voxels and more with up to 32 channels: ragged
    strips, CTAs that begin in the middle of a strip, rows too long for the
    slab (256).  Against FP64 sums of the same BF16 products, exact in FP32:
    the accumulation of n products in FP32, random in sign, is within a few
    sqrt(n) roundings; 1e-5 of the norm holds with a margin of ten."""
    import torch
    from diff_solver_b200 import _native as N
    L = N.lib()
    nx, ny, nz = shape
    assert nx * ny * nz * batch >= 30000
    g = torch.Generator(device="cpu").manual_seed(3 * cin + cout + nx)
    x = torch.randn(batch, nz, ny, nx, cin, generator=g).to(torch.bfloat16).cuda()
    dy = torch.randn(batch, nz, ny, nx, cout, generator=g).to(torch.bfloat16).cuda()
    padded = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    want = torch.stack([torch.einsum("bzyxi,bzyxo->oi", padded[:, dz:dz + nz, ddy:ddy + ny, dx:dx + nx], dy.double())
                        for dz, ddy, dx in itertools.product(range(3), repeat=3)])
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.full((L.xs_conv3d_weight_grad_scratch_floats(batch, nx, ny, nz, cin, cout),), float("nan"), device="cuda")
    dw = torch.full((27, cout, cin), 2.0, dtype=torch.float32, device="cuda")
    for accumulate in (0, 1):
        N.check("wgrad", L.xs_conv3d_weight_grad_bf16(None, batch, nx, ny, nz, cin, cout, x.data_ptr(), dy.data_ptr(), scratch.data_ptr(),
                                                      dw.data_ptr(), accumulate, err.data_ptr()))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert float((dw.double() / 2.0 - want).norm() / want.norm()) < 1e-5
