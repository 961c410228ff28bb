"""The convolution kernels of the learned correction where their tiling can go wrong: one level and an odd
level of a pair, rows that end inside a tile, more tiles than resident blocks, level chunks with a rest,
outputs that are not 16-byte aligned; and the corrected step where the first layer packs the state itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("mma", (16, 5, 1), 32, 32),      # one level a block
         ("mma", (32, 21, 33), 32, 32),    # two levels a block, the last of one; rows end inside a tile
         ("mma", (32, 21, 33), 32, 8),
         ("mma", (32, 24, 32), 16, 32),    # two levels a block
         ("mma", (32, 24, 32), 32, 16),
         ("mma", (48, 43, 33), 32, 32),    # tiles in turn on the resident blocks
         ("mma", (48, 43, 33), 16, 8),
         ("tcgen05", (16, 16, 1), 32, 32),
         ("tcgen05", (16, 16, 37), 16, 32),
         ("tcgen05", (64, 64, 45), 32, 32),   # chunks of levels with a rest
         ("tcgen05", (64, 64, 45), 32, 8),
         ("tcgen05", (112, 64, 7), 32, 16)]


@pytest.fixture
def kernel(built_lib):
    import ctypes

    def use(name):
        assert built_lib.lexgb_cnn_set_kernel({"mma": 1, "tcgen05": 2}[name]) == 0
        return built_lib
    yield use
    n = ctypes.c_uint(0)
    assert built_lib.lexgb_cnn_take_timeouts(ctypes.byref(n)) == 0
    built_lib.lexgb_cnn_set_kernel(0)
    assert n.value == 0, n.value


# tcgen05 takes 16-byte aligned outputs, mma.sync any
SHIFTS = [(k, d, a, b, s) for k, d, a, b in CASES for s in ((0, 1) if k == "mma" else (0,))]


@pytest.mark.parametrize("name,dims,cin,cout,shift", SHIFTS,
                         ids=["%s-%dx%dx%d-%d-%d-%d" % ((k,) + d + (a, b, s)) for k, d, a, b, s in SHIFTS])
def test_convolution_at_the_edges_of_its_tiles(kernel, name, dims, cin, cout, shift):
    """Against the FP64 convolution of the same BF16 operands: 27 cin products and a bias summed in FP32, in
    any order and with truncating additions, are within (27 cin + 1) 2^-23 of the sum of their magnitudes;
    the BF16 output is the GELU of that within its own error (slope at most 1.13, 2^-8 for the rounding and
    2^-10 of |x| + 1 for the hardware tanh)."""
    torch = pytest.importorskip("torch")
    import torch.nn.functional as F
    from lex_gb300 import sgs_cnn
    lib = kernel(name)
    nx, ny, nz = dims
    n = nx * ny * nz
    g = torch.Generator(device="cpu").manual_seed(cin + cout + nz)
    x = torch.randn(n, cin, generator=g).cuda().bfloat16()
    w = (torch.randn(27, cout, cin, generator=g) * 0.06).cuda().bfloat16()
    b = torch.randn(cout, generator=g).cuda()
    pre = torch.full((n * cout + 8,), float("nan"), device="cuda")
    y = torch.full((n * cout + 8,), float("nan"), device="cuda", dtype=torch.bfloat16)
    pre_v, y_v = pre[shift:shift + n * cout], y[2 * shift:2 * shift + n * cout]
    p = sgs_cnn._p
    assert lib.lexgb_cnn_conv3d(nx, ny, nz, cin, cout, p(x), p(w), p(b), p(pre_v), p(y_v), None, 1, cout,
                                sgs_cnn._stream()) == 0
    torch.cuda.synchronize()

    def conv(x, w, b):
        a = x.double().reshape(nz, ny, nx, cin).permute(3, 0, 1, 2).unsqueeze(0)
        k = w.double().reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2)
        return F.conv3d(a, k, b.double(), padding=1)[0].permute(1, 2, 3, 0).reshape(n, cout)
    ref, mag = conv(x, w, b), conv(x.abs(), w.abs(), b.abs())
    err = (27 * cin + 1) * 2.0 ** -23 * mag
    got = pre_v.view(n, cout).double()
    assert bool(((got - ref).abs() <= err).all()), float(((got - ref).abs() / err).max())
    act = F.gelu(ref, approximate="tanh")
    tol = 1.13 * err + 2.0 ** -8 * act.abs() + 2.0 ** -10 * (ref.abs() + 1)
    ya = y_v.view(n, cout).double()
    assert bool(((ya - act).abs() <= tol).all()), float(((ya - act).abs() / tol).max())
    for buf, lo in ((pre, shift), (y, 2 * shift)):   # nothing beside the output
        assert bool(buf[:lo].isnan().all()) and bool(buf[lo + n * cout:].isnan().all())


# one level, two; a plane ring that goes round (and whose first planes are held twice) within an item and
# over several items of a block; tiles that the grid does not fill
DW_DIMS = [(8, 16, 1), (8, 16, 2), (8, 16, 7), (16, 16, 150), (64, 48, 61), (20, 13, 23)]


@pytest.mark.parametrize("cin,cout,gstride", [(32, 32, 32), (16, 32, 32), (32, 8, 16)])
@pytest.mark.parametrize("dims", DW_DIMS, ids=str)
def test_weight_gradient_at_the_edges_of_its_chunks(kernel, dims, cin, cout, gstride):
    """Against the FP64 sums of the same BF16 products: at most 2 npts additions in FP32, in any order and with
    truncation, are within npts 2^-22 of the sum of their magnitudes."""
    torch = pytest.importorskip("torch")
    from lex_gb300 import sgs_cnn
    lib = kernel("tcgen05")
    nx, ny, nz = dims
    n = nx * ny * nz
    gen = torch.Generator(device="cpu").manual_seed(n + cin)
    x = torch.randn(n, cin, generator=gen).cuda().bfloat16()
    g = torch.randn(n, gstride, generator=gen).cuda().bfloat16()
    dw = torch.zeros(27, cout, cin, device="cuda")
    p = sgs_cnn._p
    assert lib.lexgb_cnn_conv3d_dw(nx, ny, nz, cin, cout, gstride, p(x), p(g), p(dw), None, sgs_cnn._stream()) == 0
    torch.cuda.synchronize()

    def sums(x, g):
        xp = torch.zeros(nz + 2, ny + 2, nx + 2, cin, device="cuda", dtype=torch.float64)
        xp[1:-1, 1:-1, 1:-1] = x.double().reshape(nz, ny, nx, cin)
        gd = g.double()[:, :cout].reshape(nz, ny, nx, cout)
        return torch.stack([torch.einsum("zyxo,zyxi->oi", gd, xp[a:a + nz, b:b + ny, c:c + nx])
                            for a in range(3) for b in range(3) for c in range(3)])
    ref, mag = sums(x, g), sums(x.abs(), g.abs())
    assert bool(((dw.double() - ref).abs() <= n * 2.0 ** -22 * mag).all())
    assert float((dw.double() - ref).norm()) <= 1e-5 * float(ref.norm())   # as the kernel's own tests


@pytest.mark.parametrize("dims", [(16, 5, 3), (32, 21, 33), (64, 64, 65)], ids=str)
def test_network_and_gradients_at_the_edges(built_lib, dims):
    """The whole network and its gradients against PyTorch, at the BF16 level of the kernels' own tests."""
    torch = pytest.importorskip("torch")
    from lex_gb300 import sgs_cnn
    from test_gpu_sgs_cnn import _reference, _rel
    n = dims[0] * dims[1] * dims[2]
    net = sgs_cnn.SGSNet(seed=1, init_scale=1.0, zero_last=False)
    for t in net.params():
        t.requires_grad_(True)
    g = torch.Generator(device="cpu").manual_seed(2)
    x = torch.rand(n, 5, generator=g).cuda().requires_grad_(True)
    out = sgs_cnn.net_apply(net, x, dims)
    xr = x.detach().clone().requires_grad_(True)
    ref, ws, bs = _reference(net, xr, dims)
    assert _rel(out.detach(), ref.detach()) < 2e-2
    seed = torch.randn(n, 5, generator=g).cuda()
    got = torch.autograd.grad((out * seed).sum(), [x] + net.params())
    want = torch.autograd.grad((ref * seed).sum(), [xr] + ws + bs)
    for i, (a, r) in enumerate(zip(got, want)):
        assert _rel(a, r.reshape(a.shape)) < 3e-2, i


@pytest.mark.parametrize("dims", [(32, 21, 33), (32, 24, 32), (16, 8, 8)], ids=str)
def test_corrected_step_equals_the_packed_network(built_lib, dims):
    """The fused correction against packing, network and unpacking one after another on the same plain step:
    the packing rounds the same way, so both feed the network the same BF16 inputs and differ by the FP32
    rounding of the addition to the state (2^-23 of a field's largest value, and as much for the product)."""
    torch = pytest.importorskip("torch")
    from lex_gb300 import autograd as lag, sgs_cnn
    from lex_gb300.solver import Solver
    from lex_gb300.workload import warm_bubble
    from test_gpu_learned_sgs import SPACING, _net_with_output
    nx, ny, nz = dims
    phys, prof = warm_bubble(nx, ny, nz, *SPACING, amplitude=2.0, radius_h=3000.0, seed=3)
    with Solver(nx, ny, nz, *SPACING, 3.0, 32, turb_opt=1) as S:
        S.integrate_base_state(prof["theta0"], prof["qv0"])
        S.upload(phys, dtype=np.float32)
        S.step(20)
        x0 = lag.get_state(S)
        S.step(10)
        scale = sgs_cnn.make_scale([x0, lag.get_state(S)])
        net = _net_with_output()
        lag.set_state(S, x0)
        S.step(1)
        plain = lag.get_state(S)
        with torch.no_grad():
            ref = sgs_cnn.correct(net, plain, scale, dims)
        sgs_cnn.attach(S, net, scale)
        lag.set_state(S, x0)
        S.step(1)
        y = lag.get_state(S)
        sgs_cnn.attach(S, None, None)
    moved = max(float((b - c).abs().max()) for b, c in zip(ref, plain))
    assert moved > 0
    for f, (a, b, c) in enumerate(zip(y, ref, plain)):
        tol = 2.0 ** -22 * float(torch.maximum(b.abs(), c.abs()).max() + (b - c).abs().max())
        assert float((a - b).abs().max()) <= tol, (f, float((a - b).abs().max()), tol)
