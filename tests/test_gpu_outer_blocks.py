"""Fronts of more pivots than one outer block of the trailing updates: separators
just past a block of 128 (1, 2, 31, 32, 33 pivots left), two whole ones and a
remainder, as single matrices (32-row tiles) and several (64-row ones where
they fill the chip), with row exchanges forced by the threshold and without.
Solutions of both orientations against SuperLU at the tolerances of the other
solves: 1e-10 relative L2 in FP64 (1e-8 where the pivots are static), 1e-8 with
complex64 factors."""
import numpy as np
import pytest

import oracle as O
from oracle import sparse as OS
from germaine_b200 import GM_PHYS_AC, GM_PREC_C64_IR, GM_PREC_FP64, GM_SYS_A, GM_SYS_AT, Engine
from tests.models import random_smooth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nf,pivot_tol", [(128, 1, 0.1), (129, 1, 1.0), (130, 6, 0.1), (159, 1, -1.0), (160, 1, 0.1),
                                             (161, 3, 1.0), (257, 1, 0.1), (263, 1, 1.0)])
def test_outer_block_remainders(ny, nf, pivot_tol):
    nx, dh, npml = ny + 9, 12.0, 5
    vp = random_smooth(nx, ny, 1700.0, 3500.0, ny)
    rho = random_smooth(nx, ny, 1000.0, 2200.0, ny + 1)
    g = O.Grid(nx=nx, ny=ny, dh=dh, npml=npml)
    freqs = np.linspace(8.0, 15.0, nf).astype(np.float32)
    rng = np.random.default_rng(ny + nf)
    b = rng.standard_normal((nf, g.n, 2)) + 1j * rng.standard_normal((nf, g.n, 2))
    last = OS.DirectSolver(OS.operator(OS.assembled_matrix(
        g, *O.Port(g).assemble(GM_PHYS_AC, float(freqs[-1]), vp, rho))))
    refs = {s: last.solve(b[-1], trans=s == GM_SYS_AT) for s in (GM_SYS_A, GM_SYS_AT)}
    for precision in (GM_PREC_FP64, GM_PREC_C64_IR):
        tol = 1e-10 if precision == GM_PREC_FP64 and pivot_tol > 0 else 1e-8
        with Engine(nx, ny, dh, npml, precision=precision, pivot_tol=pivot_tol) as e:
            e.set_model(vp, rho)
            e.factor(freqs)
            for sys, ref in refs.items():
                x = e.solve(b, sys)
                assert e.stats()["ir_residual"] <= 1e-10
                assert np.linalg.norm(x[-1] - ref) / np.linalg.norm(ref) <= tol


@pytest.mark.parametrize("nx,ny,leaf,nf", [(97, 90, 20, 1), (131, 64, 16, 2), (200, 61, 27, 12), (75, 190, 9, 3)])
def test_contribution_tiles(nx, ny, leaf, nf):
    """Contribution blocks gathered by the product's own kernel: rings that end
    inside a 32- and a 64-row tile, fronts with one child and with two, one
    matrix (32-row tiles) and several; the last matrix against SuperLU."""
    dh, npml = 11.0, 3
    vp = random_smooth(nx, ny, 1700.0, 3500.0, nx)
    rho = random_smooth(nx, ny, 1000.0, 2200.0, ny)
    g = O.Grid(nx=nx, ny=ny, dh=dh, npml=npml)
    freqs = np.linspace(7.0, 14.0, nf).astype(np.float32)
    rng = np.random.default_rng(nx + nf)
    b = rng.standard_normal((nf, g.n, 2)) + 1j * rng.standard_normal((nf, g.n, 2))
    ds = OS.DirectSolver(OS.operator(OS.assembled_matrix(
        g, *O.Port(g).assemble(GM_PHYS_AC, float(freqs[-1]), vp, rho))))
    for precision, tol in ((GM_PREC_FP64, 1e-10), (GM_PREC_C64_IR, 1e-8)):
        with Engine(nx, ny, dh, npml, precision=precision, leaf_max=leaf) as e:
            e.set_model(vp, rho)
            e.factor(freqs)
            for sys in (GM_SYS_A, GM_SYS_AT):
                ref = ds.solve(b[-1], trans=sys == GM_SYS_AT)
                x = e.solve(b, sys)
                assert e.stats()["ir_residual"] <= 1e-10
                assert np.linalg.norm(x[-1] - ref) / np.linalg.norm(ref) <= tol
