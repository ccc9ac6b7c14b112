"""40-column substitution slices above pruned 32-column ones in complex128,
which by default only a tuned table asks for.  GM_SOLVE_B=5 is read once per
process, so the solves run in a child process: shots modelled before and after
a dense solve of large values in the same buffers give the same bytes, and the
dense solution matches SuperLU (1e-10, as the other solves)."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import json
import numpy as np
import oracle as O
from oracle import sparse as OS
from germaine_b200 import GM_PHYS_AC, GM_SYS_A, GM_SYS_AT, Engine
from tests.models import random_smooth
nx, ny, dh, npml = 121, 83, 10.0, 5
vp = random_smooth(nx, ny, 1700.0, 3500.0, nx)
rho = random_smooth(nx, ny, 1000.0, 2200.0, ny)
g = O.Grid(nx=nx, ny=ny, dh=dh, npml=npml)
ds = OS.DirectSolver(OS.operator(OS.assembled_matrix(g, *O.Port(g).assemble(GM_PHYS_AC, 14.0, vp, rho))))
rx = np.arange(10, nx - 10, 3, dtype=np.int32)
ry = np.full(rx.size, 11, np.int32)
out = []
with Engine(nx, ny, dh, npml) as e:
    e.set_model(vp, rho)
    e.factor([14.0])
    for ns in (33, 37, 64, 72, 100):
        # the first shots at the top, the others at the bottom: their slices prune differently
        sx = np.linspace(20, nx - 20, ns).astype(np.float32) * dh
        sy = np.where(np.arange(ns) < 32, 12, ny - 20).astype(np.float32) * dh
        rng = np.random.default_rng(ns)
        b = 1e9 * (rng.standard_normal((g.n, ns)) + 1j * rng.standard_normal((g.n, ns)))
        first = e.forward(sx, sy, rx, ry, want_field=True)
        errs = [float(np.linalg.norm(e.solve(b, s) - r) / np.linalg.norm(r))
                for s, r in ((GM_SYS_A, ds.solve(b)), (GM_SYS_AT, ds.solve(b, trans=True)))]
        again = e.forward(sx, sy, rx, ry, want_field=True)
        same = all(bool(np.array_equal(u, v)) and float(np.abs(u).max()) > 0 for u, v in zip(first, again))
        out.append([same, max(errs)])
print(json.dumps(out))
"""


def test_pruned_forty_column_slices_in_fp64():
    env = dict(os.environ, GM_SOLVE_B="5", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert len(out) == 5
    for same, err in out:
        assert same and err <= 1e-10
