"""Static pivots of operators so small that the square of the pivot tolerance
underflows to zero (complex64: max |A| below about 4e-17; FP64: 1e-149): a zero
pivot is found by its magnitude, replaced and counted, in every factorisation
kernel, as on the same operator at unit scale."""
import numpy as np
import pytest

from germaine_b200 import GM_PREC_C64_IR, GM_PREC_FP64, Engine, _lib
from tests.test_symbolic import symbolic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pivot_tol", [0.1, -1.0])
@pytest.mark.parametrize("precision,scale", [(GM_PREC_C64_IR, 1.0), (GM_PREC_C64_IR, 1e-18), (GM_PREC_FP64, 1.0),
                                             (GM_PREC_FP64, 1e-152)])
@pytest.mark.parametrize("nx,ny", [(6, 5), (23, 17), (40, 33), (90, 30), (161, 130)])
def test_zero_pivot_is_counted_at_every_scale(nx, ny, precision, scale, pivot_tol):
    """A diagonal operator whose very last pivot is zero (nothing after it is
    touched by its reciprocal, which overflows at the small scales)."""
    S = symbolic(nx, ny, 32)
    root = int(np.nonzero(S["parent"] < 0)[0][0])
    last = int(S["vars"][S["var_off"][root] + S["npiv"][root] - 1])
    re, im = np.zeros((9, nx * ny)), np.zeros((9, nx * ny))
    re[4], im[4] = scale, -0.5 * scale
    re[4, last], im[4, last] = 0.0, 0.0
    lib = _lib.load()
    with Engine(nx, ny, 10.0, 1, precision=precision, pivot_tol=pivot_tol) as e:
        rc = lib.gm_factor_values(e._h, 1, _lib.ptr(re), _lib.ptr(im))
        assert rc == _lib.GM_WARNING_PERTURBED
        assert e.stats()["perturbed_pivots"] == 1
