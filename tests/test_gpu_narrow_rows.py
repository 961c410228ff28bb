"""The row forms of the acoustic sub-step and the short chunks of the WENO marches at their edges.

A thread of the sub-step kernel owns 4, 2 or 1 x points (nx a multiple of 4, of 2, or odd), in 16 x 4
/ 16 x 8 / 32 x 4 tiles where those fill the rows and in runs of consecutive points where they do not;
the WENO marches take chunks of 1 .. nz levels.  One step (Smagorinsky and Coriolis on) against the
FP64 oracle, to the bound of the other parity tests: 1e-5 of the increment plus the FP32 storage floor.
"""
import pytest

from test_gpu_parity import FIELDS, state_err

pytestmark = pytest.mark.gpu

#        runs of float4     full float4 tiles  float2 runs    float2 tiles   odd rows       odd rows, 32-wide
GRIDS = [(12, 7, 6), (60, 5, 9), (64, 6, 7), (128, 9, 8), (6, 9, 6), (34, 5, 11), (66, 4, 13), (5, 4, 6), (33, 6, 10)]


@pytest.mark.parametrize("dims", GRIDS, ids=lambda d: "x".join(map(str, d)))
def test_step_matches_oracle_on_row_edges(built_lib, dims):
    import numpy as np
    from oracle.dycore import Dycore
    from oracle.ic import Grid, WarmBubble, random_state
    from lex_gb300.solver import Solver
    nx, ny, nz = dims
    dx, dy, dz, dt = 600.0, 500.0, 300.0, 3.0
    phys, base, _ = WarmBubble(nx, ny, nz, dx, dy, dz).build()
    cols = dict(theta0=base[2][0, 0], qv0=base[4][0, 0], pi0=base[3][0, 0], rho0=base[1][0, 0])
    x0 = random_state(phys, nx, ny, nz, 11)
    with Solver(nx, ny, nz, dx, dy, dz, dt, 32, turb_opt=1) as S:
        S.set_base_columns(cols["theta0"], cols["qv0"], cols["pi0"], cols["rho0"])
        S.upload(x0)
        S.step(1)
        out = S.download()
    ref, _ = Dycore(Grid(nx, ny, nz, dx, dy, dz), cols, dt, 32).step(x0)
    for f, p, q, r0 in zip(FIELDS, out, ref, x0):
        assert np.isfinite(p).all()
        err = state_err(p, q, r0, f)
        assert err <= 1e-5, (f, err)
