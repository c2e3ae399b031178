"""Accuracy of the device LU's solution beside LAPACK's."""
import ctypes

import numpy as np
import pytest
import scipy.linalg as sl

from rigidfibers_kth_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,systems", [(900, 8), (2500, 3)])
def test_error_of_the_solution(n, systems):
    """Against the solution refined in extended precision.  Both factor in panels
    and sum a panel's products before they are taken off the rest, so that the
    errors are of one size: within a half of LAPACK's in the mean (one system's
    varies by a tenth)."""
    err = []
    for seed in range(systems):
        rng = np.random.default_rng(seed)
        A = np.asfortranarray(rng.normal(size=(n, n)) / np.sqrt(n) + 2 * np.eye(n))
        b, x, info = rng.normal(size=n), np.zeros(n), ctypes.c_int32(-1)
        dp = ctypes.POINTER(ctypes.c_double)
        L.check(L.lib().rf_dgesv(n, A.ctypes.data_as(dp), n, b.ctypes.data_as(dp), x.ctypes.data_as(dp), None,
                                 ctypes.byref(info), 0))
        assert info.value == 0
        lu = sl.lu_factor(A)
        lapack = sl.lu_solve(lu, b)
        ref, Al = lapack.astype(np.longdouble), A.astype(np.longdouble)
        for _ in range(3):
            ref = ref + sl.lu_solve(lu, (b - Al @ ref).astype(np.float64))
        err.append([float(np.sqrt(((v - ref) ** 2).sum() / (ref ** 2).sum())) for v in (x, lapack)])
    ours, theirs = np.mean(err, 0)
    print("n %d: %.2e, LAPACK %.2e" % (n, ours, theirs))
    assert ours <= 1.5 * theirs
