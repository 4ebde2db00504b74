"""Block GMRES with right-hand sides that stop early: a right-hand side reads only the basis vectors of its own solve.

The vectors beyond them hold whatever the plan's last solve left there, here NaN (of a solve with a NaN source).  The
right-hand sides: one that is solved before the first step (zero source), one that stops at the first vectors (a weak
source) and one that runs on; their fields are those of a fresh plan, bit for bit.
"""
import numpy as np
import pytest

from _cases import EPS_BG, WL, bead, configs, periodic, random_field
from oracle import cbs_oracle as O

import fmcuda as F

pytestmark = pytest.mark.gpu

GRID = (16, 8, 8)


def plan_of(precision):
    ocfg, solver = configs(GRID, periodic(), precision=precision, linear_solver=F.KrylovJL_GMRES(ortho="block"))
    pot = O.build_potential(ocfg, bead(GRID, 2.0), EPS_BG, WL)
    plan = solver.plan()
    plan.set_potential(pot.V, pot.k_bg, pot.eps_imag, WL)
    return solver, plan


def sources():
    S = np.zeros(GRID + (3, 3), dtype=complex, order="F")
    S[..., 1] = random_field(GRID + (3,), 1) * 1e9  # its residual meets the absolute tolerance within a few vectors
    S[..., 2] = random_field(GRID + (3,), 2) * 1e14  # (in units of k^2)
    return S


def block_solve(solver, plan):
    o = solver.solve_options(1)
    o.maxiters, o.reltol, o.abstol = 40, 1e-5, 1e-6
    return plan.solve_source(sources(), o)


@pytest.mark.parametrize("precision", ["float32-math64", "float64", "float32"])
def test_stopped_rhs_reads_its_own_vectors(precision):
    solver, plan = plan_of(precision)
    E0, H0, info0, _ = block_solve(solver, plan)
    assert np.isfinite(E0).all() and not E0[..., 0].any()
    assert 0 == info0[0].iterations < info0[1].iterations < info0[2].iterations
    solver.release()
    solver, plan = plan_of(precision)
    o = solver.solve_options(1)
    o.ortho, o.maxiters = 1, 110  # classical Gram-Schmidt fills 111 vectors of each right-hand side
    plan.solve_source(np.full_like(sources(), np.nan), o)
    E, H, info, _ = block_solve(solver, plan)
    assert [i.iterations for i in info] == [i.iterations for i in info0]
    assert np.array_equal(E, E0) and np.array_equal(H, H0)
    solver.release()
