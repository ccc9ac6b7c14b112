"""Diagonal-block factorisation and tile choice of the blocked levels: pivot
blocks of every remainder of the 8-pivot panels (1, 7, 8, 9, 31, 32 pivots
after the last full block), with row exchanges forced by the threshold and
without them, on one matrix (32-row tiles everywhere) and on eight (64-row
tiles where they fill the chip).  Both orientations against SuperLU at the
tolerances of the other solves (1e-10 relative L2; the direct solve without
exchanges is only asked to meet the refined residual)."""
import numpy as np
import pytest

import oracle as O
from oracle import sparse as OS
from germaine_b200 import GM_PHYS_AC, GM_SYS_A, GM_SYS_AT, Engine
from tests.models import random_smooth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nf", [(97, 1), (103, 1), (72, 1), (105, 8), (63, 8), (64, 1)])
@pytest.mark.parametrize("pivot_tol", [0.1, 1.0, -1.0])
def test_pivot_block_remainders(ny, nf, pivot_tol):
    nx, dh, npml = ny + 33, 12.0, 5
    vp = random_smooth(nx, ny, 1700.0, 3500.0, ny)
    rho = random_smooth(nx, ny, 1000.0, 2200.0, ny + 1)
    g = O.Grid(nx=nx, ny=ny, dh=dh, npml=npml)
    freqs = np.linspace(8.0, 15.0, nf).astype(np.float32)
    rng = np.random.default_rng(ny + nf)
    b = rng.standard_normal((nf, g.n, 3)) + 1j * rng.standard_normal((nf, g.n, 3))
    with Engine(nx, ny, dh, npml, pivot_tol=pivot_tol) as e:
        e.set_model(vp, rho)
        e.factor(freqs)
        if pivot_tol == 1.0:
            assert e.stats()["pivot_swaps"] > 0
        xs = [e.solve(b, s) for s in (GM_SYS_A, GM_SYS_AT)]
        assert e.stats()["ir_residual"] <= 1e-10
    for i in (0, nf - 1):
        ds = OS.DirectSolver(OS.operator(OS.assembled_matrix(
            g, *O.Port(g).assemble(GM_PHYS_AC, float(freqs[i]), vp, rho))))
        for x, t in zip(xs, (False, True)):
            ref = ds.solve(b[i], trans=t)
            assert np.linalg.norm(x[i] - ref) / np.linalg.norm(ref) <= (1e-10 if pivot_tol > 0 else 1e-8)
