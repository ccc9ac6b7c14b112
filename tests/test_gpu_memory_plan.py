"""gm_memory_estimate's bytes of a shot hold for the solve that takes most: one
whose refinement runs a sweep (its pivot workspace included), in both
precisions."""
import numpy as np
import pytest
import torch

from germaine_b200 import GM_PREC_C64_IR, GM_PREC_FP64, Engine
from germaine_b200.synthetic import thrust_model

pytestmark = pytest.mark.gpu

SLACK = 24 << 20   # a dozen buffers rounded up to 2 MB each


@pytest.mark.parametrize("precision", [GM_PREC_FP64, GM_PREC_C64_IR])
def test_a_refined_block_stays_within_the_estimate(precision):
    """4 matrices x 150 shots on 841 x 227 (pivot workspace: 88 MB in FP64), a
    target no solve meets and one sweep allowed."""
    nf, ns = 4, 150
    vp, rho = thrust_model(801, 187, 25.0, 20, seed=3)
    sx = np.linspace(50, 19950, ns).astype(np.float32)
    sy = np.full(ns, 50.0, np.float32)
    rx, ry = np.array([100], np.int32), np.array([2], np.int32)
    with Engine(841, 227, 25.0, 20, precision=precision, ir_tol=1e-30, ir_max_iter=1, refine=1) as e:
        e.set_model(vp, rho)
        e.factor(np.linspace(3.0, 9.0, nf).astype(np.float32))
        e.forward(sx[:1], sy[:1], rx, ry)
        free0 = torch.cuda.mem_get_info()[0]
        e.forward(sx, sy, rx, ry)
        used = free0 - torch.cuda.mem_get_info()[0]
        assert e.stats()["ir_iterations"] == 1
        _, per_shot = e.memory_estimate(nf)
        assert used <= ns * per_shot + SLACK
        assert used >= (ns - 1) * per_shot - SLACK
