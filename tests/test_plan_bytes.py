"""fm_plan_bytes counts the table of modified Gram-Schmidt that an FP64 plan holds per right-hand side (128 x 128 complex
values), which on the smallest grids is more than the fields."""
import ctypes

import pytest

from fmcuda import _lib


@pytest.mark.parametrize("precision,table", [(_lib.FM_PREC_F64, 128 * 128 * 16), (_lib.FM_PREC_F32, 0),
                                             (_lib.FM_PREC_F32_MATH64, 0)])
@pytest.mark.parametrize("nrhs", [1, 64])
def test_plan_bytes_counts_the_orthogonalisation_table(precision, table, nrhs):
    d = _lib.fm_plan_desc()
    d.grid[:], d.pad[:], d.resolution[:] = (8, 8, 8), (0, 0, 4), (50e-9,) * 3
    d.precision, d.max_rhs = precision, nrhs
    n, esz = 8 * 8 * 16, 16 if precision == _lib.FM_PREC_F64 else 8
    fields = 3 * n * esz * nrhs * (101 + 6) + n * esz + 4 * 3 * n * 16 * nrhs
    assert _lib.lib().fm_plan_bytes(ctypes.byref(d), nrhs, 101) == fields + table * nrhs
