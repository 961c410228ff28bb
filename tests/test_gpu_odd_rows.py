"""Rows of other lengths than multiples of 4 keep their arithmetic, bit for bit.

An adjoint jumps where a mass flux changes sign, so a last bit of the state that comes out otherwise shows
in a gradient, and in FP64 host output.  tests/golden/odd_rows.npz holds FP32 states (device layout, theta
relative to theta_ref) before and after one step, recorded on a GB300 from the kernels that served these
rows first: one cell a thread in the acoustic sub-step, boxes with a 3-D halo in the WENO tendencies.  Odd
rows and rows of an even length, with Coriolis (both forms), with and without the Smagorinsky tendencies.
"""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

GRIDS = [(37, 13, 12, 1, 1), (18, 11, 14, 0, 2), (21, 9, 7, 1, 0)]   # nx, ny, nz, turb_opt, cor_opt
DX, DZ, DT = 300.0, 150.0, 2.0


def make_solver(g, cols):
    from lex_gb300.solver import Solver
    nx, ny, nz, turb, cor = g
    S = Solver(nx, ny, nz, DX, DX, DZ, DT, 32, turb_opt=turb, cor_opt=cor)
    S.set_base_columns(*cols)
    return S


def one_step(g, cols, x):
    import torch
    from lex_gb300 import autograd as lag
    with make_solver(g, cols) as S:
        lag.set_state(S, [torch.from_numpy(a).cuda() for a in x], raw=True)
        S.step(1)
        return [t.cpu().numpy() for t in lag.get_state(S, raw=True)]


@pytest.mark.parametrize("g", GRIDS, ids=lambda g: "x".join(map(str, g[:3])))
def test_step_keeps_its_bits(built_lib, g):
    z = load_golden("odd_rows.npz")
    name = "x".join(map(str, g[:3]))
    y = one_step(g, [z["%s_col%d" % (name, i)] for i in range(4)], [z["%s_x%d" % (name, i)] for i in range(6)])
    for i, a in enumerate(y):
        b = z["%s_y%d" % (name, i)]
        assert a.dtype == b.dtype and np.array_equal(a, b), (i, float(np.mean(a != b)), float(np.abs(a - b).max()))
