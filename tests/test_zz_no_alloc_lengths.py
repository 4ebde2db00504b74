"""fm_green_apply_noalloc where its tables and passes change with the length: every power of two on y and z, with and
without the absorbing z boundary, and complex64 buffers that start 8 bytes off the 16 that the tile copies need (the
register passes take them, on tables of their own).

Against fm_green_apply (plan, host buffers), with the tolerances of the other operator tests.
"""
import ctypes

import numpy as np
import pytest

from _cases import EPS_BG, WL, absorbing_z, bead, configs, periodic, random_field, rel
from oracle import cbs_oracle as O

from fmcuda import _lib

pytestmark = pytest.mark.gpu

TOL = {"float64": 1e-12, "float32": 2e-6, "float32-math64": 2e-7}


@pytest.mark.parametrize("precision,shift", [("float64", 0), ("float32", 0), ("float32-math64", 0), ("float32", 1),
                                             ("float32-math64", 1)])
@pytest.mark.parametrize("padded,kind", [((16, 256, 16), "per"), ((8, 512, 8), "per"), ((32, 8, 64), "absz"),
                                         ((16, 16, 128), "absz"), ((16, 8, 256), "absz"), ((16, 8, 64), "per"),
                                         ((16, 16, 256), "per"), ((16, 8, 512), "per"), ((16, 256, 128), "absz")])
def test_noalloc_lengths(precision, shift, padded, kind):
    torch = pytest.importorskip("torch")
    grid = padded if kind == "per" else padded[:2] + (padded[2] // 2,)
    bcs = absorbing_z(grid[2]) if kind == "absz" else periodic()
    ocfg, solver = configs(grid, bcs, precision=precision)
    assert tuple(ocfg.padded_size) == padded
    pot = O.build_potential(ocfg, bead(grid, min(grid) / 4), EPS_BG, WL)
    plan = solver.plan()
    plan.set_potential(pot.V, pot.k_bg, pot.eps_imag, WL)
    x = random_field(padded + (3, 1), 5)
    ref = plan.green_apply(x)
    dt = np.complex128 if precision == "float64" else np.complex64
    n = x.size
    xd = torch.zeros(n + shift, dtype=torch.complex128 if precision == "float64" else torch.complex64, device="cuda")
    yd = torch.zeros_like(xd)
    xd[shift:] = torch.from_numpy(np.ascontiguousarray(x.astype(dt).ravel(order="F"))).cuda()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    lib = _lib.lib()
    st = lib.fm_green_apply_noalloc(ctypes.byref(plan.desc), pot.k_bg, pot.eps_imag, 1,
                                    ctypes.c_void_p(xd[shift:].data_ptr()), ctypes.c_void_p(yd[shift:].data_ptr()),
                                    stream)
    assert st == _lib.FM_OK, lib.fm_last_error().decode()
    assert rel(yd[shift:].cpu().numpy().reshape(padded + (3, 1), order="F"), ref) < TOL[precision]
    solver.release()
