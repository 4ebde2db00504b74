"""The passes at axis lengths of 128 to 512 points against the oracle, single applications (tolerances as in the other
operator tests)."""
import numpy as np
import pytest

from _cases import EPS_BG, WL, absorbing_z, bead, configs, periodic, random_field, rel
from oracle import cbs_oracle as O

pytestmark = pytest.mark.gpu


# The averaged z pass that keeps all components in registers (nz 128, 256, 512), the y tiles of 256 and 512 points and
# the row passes at those lengths: one application each against the oracle, several right-hand sides (the persistent
# CTAs of the z pass walk over right-hand sides), and nx at and off a multiple of the tile (the fallback passes).
@pytest.mark.parametrize("precision", ["float64", "float32", "float32-math64"])
@pytest.mark.parametrize("grid", [(8, 8, 64), (16, 16, 64), (12, 8, 64), (16, 8, 128), (8, 16, 256), (512, 8, 16),
                                  (16, 512, 16), (32, 256, 8), (256, 16, 16)])
def test_long_axis_passes(grid, precision):
    tol = {"float64": 1e-12, "float32": 2e-6, "float32-math64": 2e-7}[precision]
    ocfg, solver = configs(grid, absorbing_z(grid[2]), precision=precision)
    pot = O.build_potential(ocfg, bead(grid, 2.0), EPS_BG, WL)
    plan = solver.plan()
    plan.set_potential(pot.V, pot.k_bg, pot.eps_imag, WL)
    xs = [random_field(ocfg.padded_size + (3,), s) for s in (71, 72, 73)]
    X = np.asfortranarray(np.stack(xs, axis=-1))
    G, A = plan.green_apply(X), plan.apply_operator(X, X, alpha=0.7, beta=0.2j)
    for b, x in enumerate(xs):
        assert rel(G[..., b], O.green_conv(x, ocfg, pot.k_square)) < tol
        assert rel(A[..., b], O.cbs_operator(x, pot.V, ocfg, pot.k_square, alpha=0.7, beta=0.2j, y=x)) < tol
    solver.release()


# One branch of the same z pass: no shift on z (periodic) and shifts on every axis (two sweeps with their ramps, the y
# ramps inside the y tiles), at its four lengths and at nx off the tile.
@pytest.mark.parametrize("precision", ["float64", "float32", "float32-math64"])
@pytest.mark.parametrize("grid,axes", [((8, 16, 64), ""), ((12, 8, 64), ""), ((16, 8, 128), ""), ((8, 8, 256), ""),
                                       ((8, 8, 512), ""), ((16, 16, 32), "xyz"), ((8, 32, 64), "yz"), ((16, 8, 128), "xz"),
                                       ((8, 8, 256), "xyz"), ((32, 64, 16), "y")])
def test_single_branch_z_pass(grid, axes, precision):
    tol = {"float64": 1e-12, "float32": 2e-6, "float32-math64": 2e-7}[precision]
    ob, fb = zip(*[(o, f) if a in axes else (p, q) for a, n in zip("xyz", grid)
                   for (_, _, o), (p, _, _), (_, _, f), (q, _, _) in
                   [(absorbing_z(n)[0], periodic()[0], absorbing_z(n)[1], periodic()[1])]])
    ocfg, solver = configs(grid, (ob, fb), precision=precision)
    pot = O.build_potential(ocfg, bead(grid, 2.0), EPS_BG, WL)
    plan = solver.plan()
    plan.set_potential(pot.V, pot.k_bg, pot.eps_imag, WL)
    xs = [random_field(ocfg.padded_size + (3,), s) for s in (81, 82)]
    G = plan.green_apply(np.asfortranarray(np.stack(xs, axis=-1)))
    for b, x in enumerate(xs):
        assert rel(G[..., b], O.green_conv(x, ocfg, pot.k_square)) < tol
    solver.release()
