"""The network's whole-pass entries against what a caller does around them."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,dims", [("mma", (32, 32, 32)), ("mma", (48, 43, 33)), ("tcgen05", (64, 64, 32))],
                         ids=["mma-pairs", "mma-resident", "tcgen05"])
def test_forward_reads_weights_that_the_kernel_before_it_wrote(built_lib, kernel, dims):
    """lexgb_cnn_adam writes the first layer's BF16 weights, and the forward pass with x NULL (the input is in
    act[0] already) follows on the same stream with nothing between: the same bits as after a wait."""
    torch = pytest.importorskip("torch")
    from lex_gb300 import _lib, sgs_cnn
    nx, ny, nz = dims
    n = nx * ny * nz
    lib, p, st = built_lib, sgs_cnn._p, sgs_cnn._stream()
    net = sgs_cnn.SGSNet(seed=3, zero_last=False)
    gen = torch.Generator(device="cpu").manual_seed(5)
    a0 = torch.zeros(n, 16)
    a0[:, :5] = torch.rand(n, 5, generator=gen)
    acts = [a0.cuda().bfloat16()] + list(torch.empty(3, n, 32, device="cuda", dtype=torch.bfloat16))
    pres = list(torch.empty(3, n, 32, device="cuda"))
    out = torch.empty(n, 5, device="cuda")
    w0, wb0 = net.w[0].clone(), net.wbf[0].clone()
    grad = torch.randn(w0.shape, generator=gen).cuda()
    m, v = torch.zeros_like(w0), torch.zeros_like(w0)

    def run(wait):
        net.w[0].copy_(w0)
        net.wbf[0].copy_(wb0)
        for t in (m, v, out, *acts[1:], *pres):
            t.zero_()
        torch.cuda.synchronize()
        _lib.check(lib.lexgb_cnn_adam(w0.numel(), p(net.w[0]), p(grad), p(m), p(v), p(net.wbf[0]), 0.05, 0.9, 0.999,
                                      1e-8, 1, st))
        if wait:
            torch.cuda.synchronize()
        _lib.check(lib.lexgb_cnn_net_forward(nx, ny, nz, None, sgs_cnn._ptrs(net.wbf), sgs_cnn._ptrs(net.b),
                                             sgs_cnn._ptrs(acts), sgs_cnn._ptrs(pres), p(out), st))
        return [t.clone() for t in (out, *acts[1:], *pres)]

    assert lib.lexgb_cnn_set_kernel({"mma": 1, "tcgen05": 2}[kernel]) == 0
    try:
        ref = run(True)
        assert not torch.equal(net.wbf[0], wb0)
        for _ in range(5):
            for a, b in zip(run(False), ref):
                assert torch.equal(a, b)
    finally:
        lib.lexgb_cnn_set_kernel(0)
        k = ctypes.c_uint(0)
        assert lib.lexgb_cnn_take_timeouts(ctypes.byref(k)) == 0 and k.value == 0


@pytest.mark.parametrize("rows,cols", [(0, 5), (7, 5), (0, 16), (7, 16), (0, 9), (3, 4)])
def test_gradient_of_an_input_with_spare_rows_or_channels(built_lib, rows, cols):
    """net_apply takes x with more rows than the grid has points and with padding channels: its gradient has
    x's shape, zero where x takes no part; without it the weights' gradients are the same."""
    torch = pytest.importorskip("torch")
    from lex_gb300 import sgs_cnn
    dims = (16, 6, 5)
    n = 16 * 6 * 5
    net = sgs_cnn.SGSNet(seed=2, zero_last=False)
    gen = torch.Generator(device="cpu").manual_seed(7)
    x5 = torch.rand(n, 5, generator=gen).cuda().requires_grad_(True)
    x5.data[:, cols:] = 0.0
    gy = torch.randn(n, 5, generator=gen).cuda()
    y = sgs_cnn.net_apply(net, x5, dims)
    ref, = torch.autograd.grad(y, x5, gy)
    x = torch.zeros(n + rows, cols, device="cuda")
    k = min(cols, 5)
    x[:n, :k] = x5.detach()[:, :k]
    x.requires_grad_(True)
    for t in net.params():
        t.requires_grad_(True)
    out = sgs_cnn.net_apply(net, x, dims)
    assert torch.equal(out, y)
    dx, dw = torch.autograd.grad(out, [x, net.w[0]], gy)
    assert dx.shape == x.shape and dx.dtype == x.dtype
    assert torch.equal(dx[:n, :k], ref[:, :k])
    dx[:n, :k] = 0.0
    assert not dx.any()
    out = sgs_cnn.net_apply(net, x.detach(), dims)
    only, = torch.autograd.grad(out, [net.w[0]], gy)
    assert torch.allclose(only, dw, rtol=1e-4, atol=1e-5 * float(dw.abs().max()))
