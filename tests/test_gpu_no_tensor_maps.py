"""Plans whose z and y passes find no tensor maps run the register passes instead of failing.

FMCUDA_NO_TMA=2 makes the library look its encoder up in vain, as an older driver would; it is read once per process, so
the operator runs in a child process and its results are compared with this process's.  Lengths of the sixteen-value z
pass, one branch and the average of two.  FP64 is held to 1e-13 (other radices, a few roundings of 1.1e-16 on sums of
512 terms), the forms that store FP32 to 1e-6 (one rounding of 6e-8 per pass and value).
"""
import os
import subprocess
import sys

import numpy as np
import pytest

from _cases import EPS_BG, RES, WL, bead, random_field, rel

import fmcuda as F

pytestmark = pytest.mark.gpu

CASES = [(nz, absorb, precision) for nz in (64, 128, 256, 512) for absorb in (True, False)
         for precision in ("float64", "float32", "float32-math64")]


def results():
    out = []
    for nz, absorb, precision in CASES:
        grid = (16, 8, nz // 2 if absorb else nz)
        bc = F.PeriodicBoundaryCondition()
        t = nz // 2 * RES[2]
        z = F.AbsorbingBoundaryCondition(t, t, 1.0, F.TanhProfile) if absorb else bc
        solver = F.ConvergentBornSolver(resolution=RES, grid_size=grid, boundary_conditions=(bc, bc, z),
                                        precision=precision)
        plan = solver.plan()
        assert plan.padded == (16, 8, nz)
        plan.build_potential(bead(grid, 3.0), EPS_BG, WL, solver.attenuation_filters(), -1)
        out.append(plan.apply_operator(random_field(plan.padded + (3,), nz)))
        solver.release()
    return out


def test_register_passes_without_tensor_maps(tmp_path):
    path = str(tmp_path / "r.npz")
    here = os.path.dirname(os.path.abspath(__file__))
    code = ("import sys; sys.path[:0] = %r; import numpy as np, test_gpu_no_tensor_maps as t; np.savez(%r, *t.results())"
            % ([here] + sys.path[:8], path))
    done = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, FMCUDA_NO_TMA="2"), cwd=here, timeout=300,
                          capture_output=True, text=True)
    assert done.returncode == 0, done.stderr[-2000:]
    with np.load(path) as child:
        for case, mine, name in zip(CASES, results(), child.files):
            assert rel(child[name], mine) < (1e-13 if case[2] == "float64" else 1e-6), case
