"""Block GMRES where the x rows do not fill their last warp: eight rows share a warp at nx = 8 and 16, and ny * nz is odd
(general lengths on y and z), so k_xf, k_xi and the chained k_xi_xf run a warp with some of its rows alone.

Against the oracle's GMRES with the bars of the other block solves: FP64 1e-10 and the oracle's iteration count, FP32
storage 1e-5.
"""
import warnings

import pytest

from _cases import EPS_BG, bead, configs, periodic, rel, xpol
from oracle import cbs_oracle as O

import fmcuda as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bar", [("float64", 1e-10), ("float32-math64", 1e-5)])
@pytest.mark.parametrize("nx", [8, 16])
def test_block_solve_with_a_ragged_last_warp(nx, precision, bar):
    grid = (nx, 9, 7)
    ocfg, solver = configs(grid, periodic(), tol=1e-4, precision=precision,
                           linear_solver=F.KrylovJL_GMRES(ortho="block", block_size=4))
    eps, (osrc, fsrc) = bead(grid, 2.0), xpol()
    ref = O.solve(ocfg, osrc, eps, EPS_BG)
    assert ref.iterations > 8  # phase one of 4 vectors and at least one chained block
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        out = F.solve(solver, fsrc, F.Medium(eps, EPS_BG))
    if precision == "float64":
        assert solver.iteration_count == ref.iterations
    assert rel(out.E, ref.E) < bar and rel(out.H, ref.H) < bar
    solver.release()
