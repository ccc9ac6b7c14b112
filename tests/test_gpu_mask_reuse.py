"""The pruning mask and its work lists are kept by the engine between calls:
calls with other shots, more and fewer of them, give the bytes of a fresh
engine (fixed summation orders)."""
import numpy as np
import pytest

from germaine_b200 import GM_PREC_C64_IR, GM_PREC_FP64, Engine
from tests.models import random_smooth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [GM_PREC_FP64, GM_PREC_C64_IR])
def test_changing_shots_on_one_engine(precision):
    nx, ny, dh, npml = 121, 83, 10.0, 5
    vp = random_smooth(nx, ny, 1700.0, 3500.0, nx)
    rho = random_smooth(nx, ny, 1000.0, 2200.0, ny)
    rx = np.arange(10, nx - 10, 3, dtype=np.int32)
    ry = np.full(rx.size, 11, np.int32)

    def shots(ns, row):
        return np.linspace(20, nx - 20, ns).astype(np.float32) * dh, np.full(ns, row * dh, np.float32)

    def engine():
        e = Engine(nx, ny, dh, npml, precision=precision)
        e.set_model(vp, rho)
        e.factor([9.0, 14.0])
        return e

    calls = [(70, 12), (1, 60), (37, 40), (100, 12), (33, 5)]
    with engine() as kept:
        for ns, row in calls:
            got, _ = kept.forward(*shots(ns, row), rx, ry)
            with engine() as fresh:
                ref, _ = fresh.forward(*shots(ns, row), rx, ry)
            assert np.abs(got).max() > 0
            assert np.array_equal(got, ref)
