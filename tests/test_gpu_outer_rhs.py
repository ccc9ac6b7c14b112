"""Right-hand sides read where they are by the first substitution: the caller's
dense b (small fronts alone and levels of more than 32 pivots, slices of every kind of remainder)
in FP64 and complex64, one solve after another in the same buffers.  Solutions
against SuperLU at the tolerances of the other solves (1e-10 in FP64, 1e-8 with
complex64 factors)."""
import numpy as np
import pytest

import oracle as O
from oracle import sparse as OS
from germaine_b200 import GM_PHYS_AC, GM_PREC_C64_IR, GM_PREC_FP64, GM_SYS_A, GM_SYS_AT, Engine
from tests.models import random_smooth

pytestmark = pytest.mark.gpu


def _model(nx, ny):
    return random_smooth(nx, ny, 1700.0, 3500.0, nx), random_smooth(nx, ny, 1000.0, 2200.0, ny)


@pytest.mark.parametrize("nx,ny,nrhs", [(9, 7, 1), (40, 25, 33), (130, 71, 7), (130, 71, 40), (60, 117, 65)])
@pytest.mark.parametrize("precision,tol", [(GM_PREC_FP64, 1e-10), (GM_PREC_C64_IR, 1e-8)])
def test_dense_right_hand_sides(nx, ny, nrhs, precision, tol):
    dh, npml = 10.0, 2
    vp, rho = _model(nx, ny)
    g = O.Grid(nx=nx, ny=ny, dh=dh, npml=npml)
    ds = OS.DirectSolver(OS.operator(OS.assembled_matrix(g, *O.Port(g).assemble(GM_PHYS_AC, 11.0, vp, rho))))
    rng = np.random.default_rng(nrhs)
    with Engine(nx, ny, dh, npml, precision=precision) as e:
        e.set_model(vp, rho)
        e.factor([11.0])
        for k, sys in enumerate((GM_SYS_A, GM_SYS_AT, GM_SYS_A)):
            b = (rng.standard_normal((g.n, nrhs)) + 1j * rng.standard_normal((g.n, nrhs))) * 10.0 ** (6 * (1 - k))
            ref = ds.solve(b, trans=sys == GM_SYS_AT)
            x = e.solve(b, sys)
            assert np.linalg.norm(x - ref) / np.linalg.norm(ref) <= tol
