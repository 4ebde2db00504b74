"""The passes at axis lengths of 128 to 512 points against the oracle, single applications (tolerances as in the other
operator tests)."""
import numpy as np
import pytest

from _cases import EPS_BG, WL, absorbing_z, bead, configs, random_field, rel
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
