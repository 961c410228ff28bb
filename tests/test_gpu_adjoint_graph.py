"""The reverse mode's passes as graphs (from their third run on) against the same passes launched one kernel
at a time: repeated runs agree bit for bit, on another stream too, and a changed constant is taken up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(nx, ny, nz):
    from lex_gb300.solver import Solver
    from lex_gb300.workload import warm_bubble
    phys, prof = warm_bubble(nx, ny, nz, 300.0, 300.0, 300.0, amplitude=2.0, radius_h=1500.0, seed=3)
    S = Solver(nx, ny, nz, 300.0, 300.0, 300.0, 1.5, 32, turb_opt=1)
    S.integrate_base_state(prof["theta0"], prof["qv0"])
    S.upload(phys, dtype=np.float32)
    S.step(3)
    return S


@pytest.mark.parametrize("dims", [(16, 12, 9), (30, 11, 8)], ids=str)
def test_repeated_reverse_passes_agree(built_lib, dims):
    torch = pytest.importorskip("torch")
    from lex_gb300 import autograd as lag
    with _solver(*dims) as S:
        x0 = lag.get_state(S)
        g = torch.Generator(device="cpu").manual_seed(1)
        seeds = [torch.randn(t.shape, generator=g).cuda() for t in x0]

        def run(cs):
            x = [t.detach().clone().requires_grad_(True) for t in x0]
            c = torch.tensor(cs, device="cuda", requires_grad=True)
            y = lag.rollout(S, x, 2, cs=c)          # the second step is kept, the first recomputed
            return list(y) + list(torch.autograd.grad(y, x + [c], grad_outputs=seeds))

        def same(a, b):
            for i, (p, q) in enumerate(zip(a[:-1], b[:-1])):
                assert torch.equal(p, q), i
            # the constant's gradient is summed in FP64 by atomic additions of the blocks' sums
            assert abs(float(a[-1] - b[-1])) <= 1e-9 * abs(float(a[-1])) + 1e-12
        first = run(0.18)
        for _ in range(4):
            same(first, run(0.18))
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            again = run(0.18)
        torch.cuda.current_stream().wait_stream(side)
        side.synchronize()
        same(first, again)
        other = run(0.25)
        assert not torch.equal(other[0], first[0]) or not torch.equal(other[6], first[6])
        for _ in range(4):
            same(other, run(0.25))
        same(first, run(0.18))


@pytest.mark.parametrize("nx,ny,nz,copies,axis", [(15, 13, 9, 4, 2), (30, 13, 9, 2, 2), (44, 13, 9, 2, 2),
                                                  (150, 5, 6, 2, 2), (16, 4, 6, 9, 1), (12, 5, 33, 10, 1)],
                         ids=["odd rows", "even rows", "rows of four", "long rows", "four rows", "five rows, high"])
def test_reverse_pass_on_periodic_copies(built_lib, nx, ny, nz, copies, axis):
    """Periodic copies side by side are the same flow, so a grid and one of `copies` times as many points in x
    or y give the same step and the same adjoint.  The kernels take one, two or four cells a thread by the
    divisors of nx, and the flux adjoints walk rows and columns in chunks by their length: the same sums, a
    contraction or an order apart (100 sub-steps of a few operations at 2^-24: 2e-5)."""
    torch = pytest.importorskip("torch")
    from lex_gb300 import autograd as lag
    n = (nx, ny, nz)
    big = (nx * copies, ny, nz) if axis == 2 else (nx, ny * copies, nz)
    with _solver(*n) as S, _solver(*big) as D:
        x0 = lag.get_state(S)
        g = torch.Generator(device="cpu").manual_seed(2)
        seeds = [torch.randn(t.shape, generator=g).cuda() for t in x0]

        def run(solver, m):
            x = [torch.cat([t.detach()] * m, axis).contiguous().requires_grad_(True) for t in x0]
            y = lag.step(solver, x)
            return list(y) + list(torch.autograd.grad(y, x, grad_outputs=[torch.cat([t] * m, axis) for t in seeds]))
        for i, (a, b) in enumerate(zip(run(S, 1), run(D, copies))):
            a, b = a.detach().double(), b.detach().double()
            for part in torch.split(b, n[2 - axis], axis):
                assert float((part - a).norm()) <= 2e-5 * float(a.norm()), i
