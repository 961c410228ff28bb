"""The acoustic sub-steps are chained by programmatic dependent launch: each
kernel's blocks start while the one before still writes.  The state after several steps has the same bits
however the steps are submitted: as graphs, launch by launch, on the legacy default stream, on a stream of
the caller's, step by step with a wait between.  Rows of float4, of float2 and odd ones (all wide enough to
keep the whole chip busy, and small enough that a sub-step is all latency)."""
import pytest

pytestmark = pytest.mark.gpu

STEPS = 6


def runs(S, x):
    import torch
    from lex_gb300 import autograd as lag
    side = torch.cuda.Stream()
    for stream in (None, side):
        for graph in (True, False):
            for wait in (False, True):
                with torch.cuda.stream(stream) if stream else torch.cuda.stream(torch.cuda.default_stream()):
                    if stream:
                        stream.wait_stream(torch.cuda.default_stream())
                    lag.set_state(S, x, raw=True)
                    for _ in range(STEPS if wait else 1):
                        S.step(1 if wait else STEPS, graph=graph)
                        if wait:
                            torch.cuda.synchronize()
                    y = lag.get_state(S, raw=True)
                torch.cuda.synchronize()
                yield (stream is not None, graph, wait), y


def state(nx, ny, nz, qv0, seed=3):
    import torch
    g = torch.Generator(device="cpu").manual_seed(seed)
    r = lambda n, s: (torch.randn(n, ny, nx, generator=g) * s).cuda()
    w = r(nz + 1, 0.5)
    w[0] = w[-1] = 0.0
    q = torch.from_numpy(qv0[1:-1]).float().cuda()[:, None, None] * (1.0 + r(nz, 0.02))
    return r(nz, 0.5), r(nz, 2.0), r(nz, 2.0), w, r(nz, 1e-4), q


def solver(nx, ny, nz):
    import numpy as np
    from lex_gb300.solver import Solver
    S = Solver(nx, ny, nz, 600.0, 600.0, 300.0, 3.0, 32, turb_opt=1)
    qv0 = 0.014 * np.exp(-(np.arange(nz + 2) - 0.5) * 300.0 / 2500.0)
    S.integrate_base_state(np.full(nz + 2, 300.0), qv0)
    return S, qv0


@pytest.mark.parametrize("dims", [(16, 16, 12), (128, 96, 40), (18, 9, 12), (102, 75, 40), (17, 9, 12), (101, 75, 40)],
                         ids=lambda d: "x".join(map(str, d)))
def test_steps_have_the_same_bits_however_submitted(built_lib, dims):
    import torch
    S, qv0 = solver(*dims)
    with S:
        ref = None
        for how, y in runs(S, state(*dims, qv0)):
            if ref is None:
                ref = y
                assert all(torch.isfinite(a).all() for a in y)
            for a, b in zip(y, ref):
                assert torch.equal(a, b), how


def test_corrected_steps_have_the_same_bits_however_submitted(built_lib):
    import torch
    from lex_gb300 import sgs_cnn
    dims = (32, 24, 32)
    S, qv0 = solver(*dims)
    with S:
        x = state(*dims, qv0)
        kelvin = (x[0] + 300.0,) + x[1:]
        scale = sgs_cnn.make_scale([kelvin])
        scale["rout"] = 0.01 * scale["rout"]
        sgs_cnn.attach(S, sgs_cnn.SGSNet(seed=4, zero_last=False), scale)
        ref = None
        for how, y in runs(S, x):
            if ref is None:
                ref = y
                assert all(torch.isfinite(a).all() for a in y)
            for a, b in zip(y, ref):
                assert torch.equal(a, b), how
