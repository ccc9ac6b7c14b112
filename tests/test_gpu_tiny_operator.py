"""Static pivots of operators so small that the square of the pivot tolerance
underflows to zero (complex64: max |A| below about 4e-17; FP64: 1e-149):
zero pivots are found by their magnitude, replaced and counted, in every
factorisation kernel, as on the same operator at unit scale."""
import numpy as np
import pytest

from germaine_b200 import GM_PREC_C64_IR, GM_PREC_FP64, Engine, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pivot_tol", [0.1, -1.0])
@pytest.mark.parametrize("precision,scale", [(GM_PREC_C64_IR, 1.0), (GM_PREC_C64_IR, 1e-18), (GM_PREC_FP64, 1.0),
                                             (GM_PREC_FP64, 1e-152)])
def test_zero_pivots_are_counted_at_every_scale(precision, scale, pivot_tol):
    """A diagonal operator with one grid line of zeros, which meets leaves,
    the pivoted and the blocked levels: as many zero pivots as points."""
    nx, ny = 161, 130
    re, im = np.zeros((9, ny, nx)), np.zeros((9, ny, nx))
    re[4], im[4] = scale, -0.5 * scale
    re[4, 61], im[4, 61] = 0.0, 0.0
    lib = _lib.load()
    with Engine(nx, ny, 10.0, 6, precision=precision, pivot_tol=pivot_tol) as e:
        rc = lib.gm_factor_values(e._h, 1, _lib.ptr(re), _lib.ptr(im))
        assert rc == _lib.GM_WARNING_PERTURBED
        found = e.stats()["perturbed_pivots"]
        # (the reciprocal of a replaced pivot overflows at the small scales and
        # is carried on: more pivots may be found there)
        assert found == nx if scale == 1.0 else found >= nx
