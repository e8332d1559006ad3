"""The standalone products of ffea_gpu_diag_spmv are taken of a vector that
is there: on a handle that solves on chip, the right-hand side."""
import ctypes

import numpy as np
import pytest

from ffea_gb300 import params as P
from tests.helpers import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("precision", [P.PRECISION_FP64, P.PRECISION_MIXED])
def test_product_of_the_right_hand_side(gpulib, variant, precision):
    """w against the FP64 product A f in node order (compared as sorted
    values: w is in the solver's row order).  An FP32 row sums about 15 blocks
    of 3 x 3, each term rounded to 6e-8 of itself: 1e-5 of the largest."""
    from ffea_gb300 import _lib as L
    from ffea_gb300.world import World
    with World([spec(radius_nm=4.0, precision=precision, epsilon=1e-6)]) as w:
        w.run(1)
        f = w.blob(0).rhs()
        n = spec(radius_nm=4.0).mesh.num_linear
        want = np.zeros_like(f)
        L.check(gpulib.ffea_gpu_solver_apply(w.handle, 0, L.ptr(f), L.ptr(want)), "apply")
        assert w.diag_spmv(variant, reps=1) > 0
        rows = ctypes.c_int32()
        L.check(gpulib.ffea_gpu_diag_cg_vectors(w.handle, 0, ctypes.byref(rows), None, None, None, None), "diag")
        got = np.zeros(3 * rows.value, np.float64 if precision == P.PRECISION_FP64 else np.float32)
        L.check(gpulib.ffea_gpu_diag_cg_vectors(w.handle, 0, ctypes.byref(rows), None, None, got.ctypes.data, None),
                "diag")
    want = want.reshape(-1, 3)[:n].reshape(-1)
    assert np.abs(want).max() > 0 and len(got) >= len(want)
    want = np.concatenate([want, np.zeros(len(got) - len(want))])  # padding rows
    tol = 1e-12 if precision == P.PRECISION_FP64 else 1e-5
    np.testing.assert_allclose(np.sort(got.astype(np.float64)), np.sort(want), rtol=0, atol=tol * np.abs(want).max())
