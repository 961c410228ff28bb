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
