"""The residual of a restart in the FP32-storage form with FP64 arithmetic, whose passes run on FP64 copies in the dead
basis vectors: cycle lengths on both sides of the room they need, odd field sizes (the copies are aligned up), one and
two Green branches, and right-hand sides that leave at different iterations (their vectors hold the copies' bytes).

Against the oracle's GMRES(m), 1e-5 as in the other solve tests of this form.
"""
import warnings

import pytest

from _cases import EPS_BG, WL, absorbing_z, bead, configs, periodic, rel
from oracle import cbs_oracle as O
from test_gpu_absorbing_xy import absorbing_on

import fmcuda as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,bcs", [((5, 7, 3), "per"), ((16, 16, 8), "z"), ((9, 8, 11), "xyz")])
@pytest.mark.parametrize("restart", [8, 9, 11, 14])
def test_restart_residual(grid, bcs, restart):
    pair = {"per": periodic(), "z": absorbing_z(grid[2]), "xyz": absorbing_on(grid, (0, 1, 2))}[bcs]
    ls = F.KrylovJL_GMRES(gmres_restart=restart)
    ocfg, solver = configs(grid, pair, tol=1e-4, precision="float32-math64", linear_solver=ls)
    eps = bead(grid, min(grid) / 3)
    waves = [([1, 0, 0], [0, 0, 1]), ([0, 1, 0], [0, 0, 1]), ([0, 1, 0], [0.6, 0, 0.8])]
    refs = [O.solve(ocfg, O.PlaneWave(WL, p, k), eps, EPS_BG, restart=restart) for p, k in waves]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        outs = F.solve_batch(solver, [[F.PlaneWaveSource(wavelength=WL, polarization=p, k_vector=k)] for p, k in waves],
                             F.Medium(eps, EPS_BG))
    for out, ref in zip(outs, refs):
        assert rel(out.E, ref.E) < 1e-5
        assert rel(out.H, ref.H) < 1e-5
    solver.release()
