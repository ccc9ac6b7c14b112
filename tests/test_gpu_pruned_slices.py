"""Pruned forward passes whose slices differ in width between the levels (32
columns on the small fronts, 40 above in complex64): the columns of a pruned
slice are not read, so a solve does not depend on what an earlier one left in
its buffers."""
import numpy as np
import pytest

from germaine_b200 import GM_PREC_C64_IR, GM_PREC_FP64, GM_SYS_A, Engine
from tests.models import random_smooth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [1, 32, 37, 64, 100])
def test_spikes_do_not_depend_on_the_buffers(ns):
    """The same shots before and after a dense solve of large values in the same
    buffers, in both precisions: equal bytes (fixed summation orders)."""
    nx, ny, dh, npml = 121, 83, 10.0, 5
    vp = random_smooth(nx, ny, 1700.0, 3500.0, nx)
    rho = random_smooth(nx, ny, 1000.0, 2200.0, ny)
    sx = np.linspace(20, nx - 20, ns).astype(np.float32) * dh
    sy = np.full(ns, 12 * dh, np.float32)
    rx = np.arange(10, nx - 10, 3, dtype=np.int32)
    ry = np.full(rx.size, 11, np.int32)
    rng = np.random.default_rng(ns)
    b = 1e9 * (rng.standard_normal((2, nx * ny, ns)) + 1j * rng.standard_normal((2, nx * ny, ns)))
    for precision in (GM_PREC_FP64, GM_PREC_C64_IR):
        with Engine(nx, ny, dh, npml, precision=precision) as e:
            e.set_model(vp, rho)
            e.factor([9.0, 14.0])
            first = e.forward(sx, sy, rx, ry, want_field=True)
            e.solve(b, GM_SYS_A)
            again = e.forward(sx, sy, rx, ry, want_field=True)
            for u, v in zip(first, again):
                assert np.all(np.isfinite(u)) and np.abs(u).max() > 0
                assert np.array_equal(u, v)
