"""Solves that store complex64 return the same fields, bit for bit, as when these digests were recorded.

Such a solve rounds every stored value, and one different bit before a rounding becomes other rounding noise in all of
the field within a few iterations: a change of a transform's radices, of the place of a rounding or of the order of a
sum moves the fields of a long solve by more than FP32 resolves (2e-5 at 512 x 64 x 512, GMRES(20)).  So the order of
the arithmetic belongs to the results.  The digests are SHA-256 of E and H as complex64, recorded on a B200 with 148
SMs (the sums over a field are split by the number of SMs) and code built by CUDA 12.9.  The cases reach each length
of the x, y and z passes whose arithmetic FP32 storage chooses apart from FP64 storage, and the general lengths.
"""
import hashlib
import json
import os
import warnings

import numpy as np
import pytest

from _cases import EPS_BG, RES, WL, bead

import fmcuda as F

pytestmark = pytest.mark.gpu

GMRES, GMRES20, BICG = F.KrylovJL_GMRES(), F.KrylovJL_GMRES(gmres_restart=20), F.KrylovJL_BICGSTAB()
CASES = {  # grid, layer of voxels per side that absorbs (z; a negative number: on all axes), precision, solver
    "x256": ((256, 16, 32), 16, "float32-math64", GMRES20),
    "x512": ((512, 16, 32), 16, "float32-math64", GMRES20),
    "y256": ((16, 256, 32), 16, "float32-math64", GMRES20),
    "y512": ((16, 512, 16), 8, "float32-math64", GMRES20),
    "z64": ((32, 32, 32), 16, "float32-math64", GMRES20),
    "z128": ((32, 32, 64), 32, "float32-math64", GMRES20),
    "z256": ((32, 32, 128), 64, "float32-math64", GMRES20),
    "z512": ((32, 32, 256), 128, "float32-math64", GMRES20),
    "z256_periodic": ((32, 32, 256), 0, "float32-math64", GMRES),
    "z512_periodic": ((32, 16, 512), 0, "float32-math64", GMRES),
    "open": ((48, 48, 48), -8, "float32-math64", GMRES),
    "single_z64": ((32, 32, 32), 16, "float32", GMRES),
    "single_z128": ((64, 64, 64), 32, "float32", GMRES),
    "single_z256": ((32, 32, 128), 64, "float32", GMRES),
    "single_z512": ((32, 32, 256), 128, "float32", GMRES),
    "single_z256_periodic": ((32, 32, 256), 0, "float32", GMRES),
    "single_bicgstab": ((32, 32, 32), 16, "float32", BICG),
    "mgs": ((64, 32, 32), 16, "float32-math64", F.KrylovJL_GMRES(gmres_restart=20, ortho="mgs")),
    "cgs2": ((32, 32, 32), 16, "float32-math64", F.KrylovJL_GMRES(ortho="cgs2")),
    "single_41x73x58": ((41, 73, 50), 4, "float32", GMRES),
    "single_51x85x51": ((51, 85, 43), 4, "float32", GMRES),
    "single_open_general": ((30, 33, 25), -5, "float32", GMRES),
    "general_66x90x99": ((66, 90, 59), 20, "float32-math64", GMRES20),
    "general_128x96x101": ((128, 96, 61), 20, "float32-math64", GMRES20),
    "general_open": ((30, 33, 25), -5, "float32-math64", GMRES),
    "general_z96": ((32, 32, 64), 16, "float32-math64", GMRES),
    "single_z96": ((32, 32, 64), 16, "float32", GMRES),
}


def digests(name):
    grid, layer, precision, linear = CASES[name]

    def absorbing():
        t = 2 * abs(layer) * RES[2]
        return F.AbsorbingBoundaryCondition(t, t, 1.0, F.TanhProfile)
    bcs = [absorbing() if layer < 0 or (layer and a == 2) else F.PeriodicBoundaryCondition() for a in range(3)]
    solver = F.ConvergentBornSolver(resolution=RES, grid_size=grid, boundary_conditions=bcs, tolerance=1e-6,
                                    iterations_max=50, precision=precision, linear_solver=linear)
    wave = F.PlaneWaveSource(wavelength=WL, polarization=[1, 0, 0], k_vector=[0, 0, 1])
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        out = F.solve(solver, wave, F.Medium(bead(grid, min(grid) / 3), EPS_BG))
    solver.release()
    return [hashlib.sha256(np.asfortranarray(a.astype(np.complex64)).tobytes(order="F")).hexdigest() for a in (out.E, out.H)]


@pytest.mark.parametrize("name", CASES)
def test_fields_are_the_recorded_ones(name):
    with open(os.path.join(os.path.dirname(__file__), "golden", "fp32_storage_bits.json")) as f:
        recorded = json.load(f)
    assert digests(name) == recorded[name]
