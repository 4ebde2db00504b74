"""The Gram-Schmidt sweeps (k_gsdot, k_gsupdate) at the edges of their tiles, against the oracle's GMRES (modified
Gram-Schmidt): fields of an odd number of values and of fewer values than one sweep step per warp, basis sizes on and
off the group of four vectors, restarts, and right-hand sides that stop at different iterations.

Tolerances as in the other solve tests: FP64 1e-10 and the oracle's iteration count, FP32 forms 1e-5.  A non-finite
input has to come back non-finite (the FP32 values are widened without the conversion instruction).
"""
import warnings

import numpy as np
import pytest

from _cases import EPS_BG, WL, absorbing_z, bead, configs, periodic, random_field, rel
from oracle import cbs_oracle as O

import fmcuda as F

pytestmark = pytest.mark.gpu

TOL = {"float64": 1e-10, "float32": 1e-5, "float32-math64": 1e-5}


@pytest.mark.parametrize("ortho,precision", [("mgs", "float64"), ("mgs", "float32-math64"), ("cgs", "float32"),
                                             ("cgs2", "float32-math64"), ("cgs", "float64")])
@pytest.mark.parametrize("grid,bcs,restart", [((5, 7, 3), "per", 0), ((8, 8, 8), "per", 5), ((16, 16, 8), "absz", 7),
                                              ((21, 10, 13), "absz", 4)])
def test_gram_schmidt_sweeps(ortho, precision, grid, bcs, restart):
    pair = absorbing_z(grid[2]) if bcs == "absz" else periodic()
    ls = F.KrylovJL_GMRES(ortho=ortho, gmres_restart=restart)
    ocfg, solver = configs(grid, pair, tol=1e-4, precision=precision, linear_solver=ls)
    eps = bead(grid, min(grid) / 3)
    waves = [([1, 0, 0], [0, 0, 1]), ([0, 1, 0], [0, 0, 1]), ([0, 1, 0], [0.6, 0, 0.8])]
    refs = [O.solve(ocfg, O.PlaneWave(WL, p, k), eps, EPS_BG, restart=restart) for p, k in waves]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        outs = F.solve_batch(solver, [[F.PlaneWaveSource(wavelength=WL, polarization=p, k_vector=k)] for p, k in waves],
                             F.Medium(eps, EPS_BG))
    for out, ref, info in zip(outs, refs, solver.last_info):
        if precision == "float64":
            assert info["iterations"] == ref.iterations
        assert rel(out.E, ref.E) < TOL[precision]
        assert rel(out.H, ref.H) < TOL[precision]
    solver.release()


@pytest.mark.parametrize("precision", ["float32", "float32-math64", "float64"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_source_stays_non_finite(precision, bad):
    grid = (8, 8, 8)
    ocfg, solver = configs(grid, periodic(), precision=precision, linear_solver=F.KrylovJL_GMRES(ortho="mgs"))
    pot = O.build_potential(ocfg, bead(grid, 2.0), EPS_BG, WL)
    plan = solver.plan()
    plan.set_potential(pot.V, pot.k_bg, pot.eps_imag, WL)
    S = random_field(grid + (3,), 3)
    S[1, 2, 3, 1] = bad
    opts = solver.solve_options(1)
    opts.maxiters = 6
    E, _, _, _ = plan.solve_source(S, opts)
    assert not np.isfinite(E).any()
    solver.release()
