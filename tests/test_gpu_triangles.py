"""Whole-triangle inverses of the fronts with more than 32 pivots: solves of
both orientations against SuperLU at the sizes where the doubling and the
32-row tiles can go wrong -- separators of 33, 64, 65, 96, 97 and 130 pivots
(one pivot over a block, full and nearly full pairs, an unpaired last
block) -- one and 33 right-hand sides, and leaves of more than 32 pivots.
Tolerances as for the other solves: relative L2 error 1e-10 in FP64, 1e-8
with complex64 factors refined to 1e-10."""
import numpy as np
import pytest

import oracle as O
from oracle import sparse as OS
from germaine_b200 import GM_PHYS_AC, GM_PREC_C64_IR, GM_PREC_FP64, GM_SYS_A, GM_SYS_AT, Engine
from tests.models import random_smooth

pytestmark = pytest.mark.gpu


def _problem(nx, ny, dh, npml):
    vp = random_smooth(nx, ny, 1800.0, 3200.0, nx + ny)
    rho = random_smooth(nx, ny, 1000.0, 2000.0, nx - ny)
    g = O.Grid(nx=nx, ny=ny, dh=dh, npml=npml)
    ds = OS.DirectSolver(OS.operator(OS.assembled_matrix(g, *O.Port(g).assemble(GM_PHYS_AC, 12.0, vp, rho))))
    return g, vp, rho, ds


@pytest.mark.parametrize("ny,leaf", [(33, 32), (64, 32), (65, 32), (96, 20), (97, 32), (130, 32), (70, 64)])
def test_triangle_inverses_solve(ny, leaf):
    nx, dh, npml = ny + 40, 10.0, 6
    g, vp, rho, ds = _problem(nx, ny, dh, npml)
    rng = np.random.default_rng(ny)
    for precision, tol in ((GM_PREC_FP64, 1e-10), (GM_PREC_C64_IR, 1e-8)):
        with Engine(nx, ny, dh, npml, precision=precision, leaf_max=leaf) as e:
            e.set_model(vp, rho)
            e.factor([12.0])
            assert e.stats()["max_piv"] == max(ny, leaf if leaf > 32 else 0)
            for nrhs in (1, 33):
                b = rng.standard_normal((g.n, nrhs)) + 1j * rng.standard_normal((g.n, nrhs))
                for sys in (GM_SYS_A, GM_SYS_AT):
                    x, ref = e.solve(b, sys), ds.solve(b, trans=sys == GM_SYS_AT)
                    err = np.linalg.norm(x - ref) / np.linalg.norm(ref)
                    assert err <= tol, f"precision {precision}, {nrhs} rhs, sys {sys}: {err:.2e}"
