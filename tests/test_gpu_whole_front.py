"""Whole-front kernel of the lower levels at the sizes where it can go wrong:
leaves of 4 .. 32 and more than 32 pivots (every remainder of the 8-pivot
panels, fronts of one to several size classes and of each thread count),
grids whose leaves reach the boundary, and the levels just below and above
the line where row exchanges begin (exchanges forced with a threshold of 1).
Residuals against the assembled operator and solutions against SuperLU, both
orientations, at the tolerances of the other solves: 1e-10 in FP64, 1e-8 with
complex64 factors."""
import numpy as np
import pytest

import oracle as O
from oracle import sparse as OS
from germaine_b200 import GM_PHYS_AC, GM_PREC_C64_IR, GM_PREC_FP64, GM_SYS_A, GM_SYS_AT, Engine
from tests.models import random_smooth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,leaf", [(7, 5, 40), (23, 17, 4), (61, 47, 9), (90, 33, 13), (57, 121, 25), (128, 96, 31),
                                        (75, 75, 33), (66, 40, 48), (80, 64, 64), (230, 30, 32)])
@pytest.mark.parametrize("pivot_tol", [0.1, 1.0])
def test_whole_front_solve(nx, ny, leaf, pivot_tol):
    dh, npml = 10.0, 2
    vp = random_smooth(nx, ny, 1700.0, 3500.0, nx)
    rho = random_smooth(nx, ny, 1000.0, 2200.0, ny)
    g = O.Grid(nx=nx, ny=ny, dh=dh, npml=npml)
    freqs = np.array([9.0, 14.0], np.float32)
    ops = [OS.DirectSolver(OS.operator(OS.assembled_matrix(g, *O.Port(g).assemble(GM_PHYS_AC, float(f), vp, rho))))
           for f in freqs]
    rng = np.random.default_rng(nx * ny)
    b = rng.standard_normal((2, g.n, 5)) + 1j * rng.standard_normal((2, g.n, 5))
    for precision, tol in ((GM_PREC_FP64, 1e-10), (GM_PREC_C64_IR, 1e-8)):
        with Engine(nx, ny, dh, npml, precision=precision, leaf_max=leaf, pivot_tol=pivot_tol) as e:
            e.set_model(vp, rho)
            e.factor(freqs)
            for sys in (GM_SYS_A, GM_SYS_AT):
                x = e.solve(b, sys)
                assert e.stats()["ir_residual"] <= 1e-10
                for i, ds in enumerate(ops):
                    ref = ds.solve(b[i], trans=sys == GM_SYS_AT)
                    assert np.linalg.norm(x[i] - ref) / np.linalg.norm(ref) <= tol


@pytest.mark.parametrize("nrhs", [1, 8, 9, 16, 17, 31, 33, 48, 100])
def test_small_front_slices(nrhs):
    """Substitution slices of the small fronts: dealt to the warps by columns
    above 16 right-hand sides and by rows up to there, fronts of every pivot
    group (leaves of 6 to 30 pivots on one grid)."""
    nx, ny, dh, npml = 101, 67, 10.0, 3
    vp = random_smooth(nx, ny, 1700.0, 3500.0, 5)
    rho = random_smooth(nx, ny, 1000.0, 2200.0, 6)
    g = O.Grid(nx=nx, ny=ny, dh=dh, npml=npml)
    ds = OS.DirectSolver(OS.operator(OS.assembled_matrix(g, *O.Port(g).assemble(GM_PHYS_AC, 11.0, vp, rho))))
    rng = np.random.default_rng(nrhs)
    b = rng.standard_normal((g.n, nrhs)) + 1j * rng.standard_normal((g.n, nrhs))
    for precision, tol in ((GM_PREC_FP64, 1e-10), (GM_PREC_C64_IR, 1e-8)):
        with Engine(nx, ny, dh, npml, precision=precision) as e:
            e.set_model(vp, rho)
            e.factor([11.0])
            for sys in (GM_SYS_A, GM_SYS_AT):
                x, ref = e.solve(b, sys), ds.solve(b, trans=sys == GM_SYS_AT)
                assert np.linalg.norm(x - ref) / np.linalg.norm(ref) <= tol
