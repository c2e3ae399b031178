"""rf_dgesv at the ends of the FP64 range, against IEEE division (numpy)."""
import ctypes

import numpy as np
import pytest

from rigidfibers_kth_b200 import _lib as L

pytestmark = pytest.mark.gpu


def dgesv(A, b):
    n = len(b)
    A = np.asfortranarray(A, dtype=np.float64)
    x, piv, info = np.zeros(n), np.zeros(n, dtype=np.int32), ctypes.c_int32(-1)
    dp = ctypes.POINTER(ctypes.c_double)
    L.check(L.lib().rf_dgesv(n, A.ctypes.data_as(dp), n, b.ctypes.data_as(dp), x.ctypes.data_as(dp), piv.ctypes.data,
                             ctypes.byref(info), 0))
    return x, piv, info.value


# the largest number, both sides of 2^1022 (where the reciprocal leaves the
# normal range), of the smallest normal number and of the lines at 2^960 and 2^-959, subnormals
ENDS = [1.7976931348623157e308, -1e308, 4.5e307, 4.4e307, 1e300, 9.8e288, 9.7e288, 3.0, -1.0, 1.1e-289, 1.0e-289,
        1e-300, 2.3e-308, -2.2e-308, 1e-308, 1e-310, 5e-324]


@pytest.mark.parametrize("d", ENDS)
def test_one_by_one(d):
    """x = b / d exactly as the division rounds it, overflow and underflow included."""
    for v in (1.0, -3.7, 0.0, 1e308, 1e300, 1e-300, 1e-308, 5e-324, 0.3 * d):
        x, _, info = dgesv(np.array([[d]]), np.array([v]))
        with np.errstate(over="ignore", under="ignore"):
            assert info == 0 and x[0] == np.float64(v) / np.float64(d)


@pytest.mark.parametrize("n,seed", [(31, 0), (130, 1), (300, 2)])
def test_diagonal(n, seed):
    """Pivots over the normal range: every row is one division."""
    rng = np.random.default_rng(seed)
    d = rng.choice([-1, 1], n) * rng.uniform(1, 10, n) * 10.0 ** rng.integers(-307, 307, n)
    d[:10] = [1e308, -1.7e308, 4.5e307, 1e300, 2.3e-308, 1e-300, 1e290, 1e-290, 3.0, -7.0]
    x0 = rng.uniform(-10, 10, n)
    with np.errstate(over="ignore", under="ignore"):
        b = np.clip(x0 * d, -1.7e308, 1.7e308)
        b[12] = 0.0
        ref = b / d
    x, piv, info = dgesv(np.diag(d), b)
    assert info == 0 and np.array_equal(piv, np.arange(1, n + 1))
    assert np.array_equal(x, ref)


@pytest.mark.parametrize("scale", [1e-300, 1e-290, 1e290, 1e300])
def test_scaled_system(scale):
    """A general system with every entry scaled: the solution is the unscaled one's
    to rounding (backward error within n units on the unscaled matrix)."""
    n = 97
    rng = np.random.default_rng(7)
    A, b = rng.standard_normal((n, n)), rng.standard_normal(n)
    x, _, info = dgesv(A * scale, b * scale)
    assert info == 0
    assert np.linalg.norm(A @ x - b) <= n * 2.0 ** -52 * np.linalg.norm(A) * np.linalg.norm(x)


@pytest.mark.parametrize("n", [2, 33, 150])
def test_subnormal_pivots(n):
    """Subnormal pivots above other rows (LAPACK's dgetf2 divides there): a lower
    triangle of ones and a diagonal, both times 2^-1050; every step is exact."""
    s = 2.0 ** -1050
    x0 = np.random.default_rng(n).integers(-8, 9, n).astype(np.float64)
    tri = np.tril(np.ones((n, n)))
    for A in (tri, np.diag(np.arange(1.0, n + 1))):
        for rows in (np.arange(n), np.arange(n)[::-1]):  # as they stand, and every pivot a swap
            x, _, info = dgesv(A[rows] * s, (A @ x0)[rows] * s)
            assert info == 0 and np.array_equal(x, x0)
