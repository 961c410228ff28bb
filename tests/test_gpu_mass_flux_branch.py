"""Forward and reverse pass take the same stencil where a mass flux vanishes.

The sign of a face's mass flux picks the WENO stencil, zero counting as upward.  Where a wind changes
sign from one point to the next at equal size, the mass flux of its own field is exactly zero; a reverse
pass that forms it with another rounding gets a residual of either sign and differentiates the stencil
the forward pass did not take.  One stage (a single sub-step) of such states, alternating along x, y or z,
against torch.autograd through the FP64 oracle: 1e-4 of each field's adjoint, the bound of the other
reverse-mode tests.  Rows of float4, of float2 and odd ones.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-4


@pytest.mark.parametrize("axis,dims", [("x", (12, 7, 9)), ("x", (14, 7, 9)), ("y", (12, 10, 9)), ("y", (13, 34, 9)),
                                       ("z", (12, 7, 9)), ("z", (9, 7, 40))],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_reverse_takes_the_forward_stencil(built_lib, axis, dims):
    import torch
    from oracle.dycore import Dycore
    from oracle.ic import Grid, WarmBubble, pad_scalar, pad_u, pad_v, random_state
    from lex_gb300.solver import Solver
    nx, ny, nz = dims
    dx, dy, dz, dt = 600.0, 500.0, 300.0, 3.0
    phys, base, _ = WarmBubble(nx, ny, nz, dx, dy, dz).build()
    cols = dict(theta0=base[2][0, 0], qv0=base[4][0, 0], pi0=base[3][0, 0], rho0=base[1][0, 0])
    x0 = random_state(phys, nx, ny, nz, 23)
    c = (slice(3, -3), slice(3, -3), slice(1, -1))
    inner = [x0[0][c], x0[1][3:3 + nx, 3:-3, 1:-1], x0[2][3:-3, 3:3 + ny, 1:-1], x0[3][c], x0[4][c], x0[5][c]]
    inner = [np.array(a, dtype=np.float32) for a in inner]
    if axis == "x":      # nx is even: every mass flux of u along x is zero
        inner[1] = inner[1][:1] * np.where(np.arange(nx) % 2, -1, 1).astype(np.float32)[:, None, None]
    elif axis == "y":
        inner[2] = inner[2][:, :1] * np.where(np.arange(ny) % 2, -1, 1).astype(np.float32)[None, :, None]
    else:                # those of w in the cells between the first and the last inner face
        inner[3][:, :, 1:-1] = inner[3][:, :, 1:2] * np.where(np.arange(nz - 1) % 2, -1, 1).astype(np.float32)
    rng = np.random.default_rng(29)
    yb = [rng.standard_normal(a.shape).astype(np.float32) * s for a, s in zip(inner, (0.3, 1, 1, 0.5, 1, 1))]
    yb[3][:, :, 0] = yb[3][:, :, -1] = 0.0

    cat = torch.cat
    leaf = [torch.from_numpy(a.astype(np.float64)).requires_grad_(True) for a in inner]
    T, u, v, w, p, q = leaf
    state = (pad_scalar(T), pad_u(cat([u, u[:1]], 0)), pad_v(cat([v, v[:, :1]], 1)), pad_scalar(w), pad_scalar(p),
             pad_scalar(q))
    D = Dycore(Grid(nx, ny, nz, dx, dy, dz), cols, dt, 32, turb=False, device="cpu")
    dts, n = D.stage_plan()[0]
    y, _ = D.stage(state, state, dts, None, n)
    y = [y[0][c], y[1][3:3 + nx, 3:-3, 1:-1], y[2][3:-3, 3:3 + ny, 1:-1], y[3][c], y[4][c], y[5][c]]
    ref = torch.autograd.grad(sum((a * torch.from_numpy(b.astype(np.float64))).sum() for a, b in zip(y, yb)), leaf)

    with Solver(nx, ny, nz, dx, dy, dz, dt, 32, turb_opt=0) as S:
        S.set_base_columns(cols["theta0"], cols["qv0"], cols["pi0"], cols["rho0"])
        S.upload([a.detach().numpy() for a in state])
        got = S.step_vjp(yb, nstages=1)
    err = []
    for f, (a, b) in enumerate(zip(got, ref)):
        k = slice(1, -1) if f == 3 else slice(None)      # w on its free faces
        a, b = a[:, :, k], b.numpy()[:, :, k]
        err.append(float(np.linalg.norm(a - b) / np.linalg.norm(b)))
    assert max(err) <= TOL, err
