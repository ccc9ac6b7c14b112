"""Row exchanges inside the one-warp panels, in the whole-front kernel's
levels (80 rows and more) and the blocked ones, whenever a larger entry exists
(threshold 1): on operators of random entries in all nine directions (rows
trade multipliers that other lanes stored a pivot before), and where the larger
entry differs from the pivot by less than the leading bits of its square
show."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import sparse as OS
from germaine_b200 import GM_OP_EXACT, GM_SYS_A, GM_SYS_AT, Engine, _lib

pytestmark = pytest.mark.gpu


def _factor(e, re, im):
    rc = _lib.load().gm_factor_values(e._h, 1, _lib.ptr(re), _lib.ptr(im))
    e.nf = 1
    return rc


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_random_operator_with_exchanges(seed):
    """Direct solves (before any refinement) and solutions against SuperLU, both
    orientations.  The numpy replay of the factorisation makes 898 to 1018
    exchanges on these operators and leaves residuals up to 5e-13 and errors up
    to 2e-13; a multiplier of another row leaves residuals near 1."""
    nx, ny = 161, 130
    n = nx * ny
    rng = np.random.default_rng(seed)
    v = rng.standard_normal((9, ny, nx)) + 1j * rng.standard_normal((9, ny, nx))
    v[4] *= 3.0
    r, c, w = [], [], []
    k = np.arange(n).reshape(ny, nx)
    for q in range(9):
        di, dj = q % 3 - 1, q // 3 - 1
        y0, y1, x0, x1 = max(0, -dj), ny - max(0, dj), max(0, -di), nx - max(0, di)
        r.append(k[y0:y1, x0:x1].ravel())
        c.append(r[-1] + di + dj * nx)
        w.append(v[q, y0:y1, x0:x1].ravel())
    M = sp.csc_matrix((np.concatenate(w), (np.concatenate(r), np.concatenate(c))), (n, n))
    ds = OS.DirectSolver(M)
    b = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    with Engine(nx, ny, 10.0, 6, op_mode=GM_OP_EXACT, pivot_tol=1.0) as e:
        assert _factor(e, np.ascontiguousarray(v.real), np.ascontiguousarray(v.imag)) >= 0
        assert e.stats()["pivot_swaps"] > 500
        for sys in (GM_SYS_A, GM_SYS_AT):
            x, ref = e.solve(b, sys), ds.solve(b, trans=sys == GM_SYS_AT)
            assert e.refine_report()[0]["first_residual"] <= 1e-11
            assert np.linalg.norm(x - ref) / np.linalg.norm(ref) <= 1e-10


def test_exchanges_by_the_last_bits():
    """Grid points coupled in pairs along y, [[1, -(1 + d)], [1 + d, 1]]: every
    pair inside one pivot block trades rows, by d = 2^-10 as by d = 2^-30 (whose
    square has the leading 32 bits of 1)."""
    nx, ny = 161, 130
    swaps = []
    for d in (2.0 ** -10, 2.0 ** -30):
        re, im = np.zeros((9, ny, nx)), np.zeros((9, ny, nx))
        re[4] = 1.0
        re[1, 1::2] = 1.0 + d     # odd lines: the entry of the line above
        re[7, 0::2] = -1.0 - d    # even lines: the entry of the line below
        with Engine(nx, ny, 10.0, 6, op_mode=GM_OP_EXACT, pivot_tol=1.0) as e:
            assert _factor(e, re, im) == _lib.GM_OK
            swaps.append(e.stats()["pivot_swaps"])
            k = np.zeros(nx * ny)
            k[::3] = 1.0
            x = e.solve(k).reshape(ny, nx)
            up, lo = x[0::2], x[1::2]
            b = k.reshape(ny, nx)
            assert np.abs(up - (1 + d) * lo - b[0::2]).max() <= 1e-14
            assert np.abs((1 + d) * up + lo - b[1::2]).max() <= 1e-14
    assert swaps[0] == swaps[1] > 0
