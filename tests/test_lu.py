"""The device LU (rf_dgesv) at the edges of its panels (128 columns), register
sub-panels (32, 16, 8 columns by the rows left: 4096, 8192, 16384, 32768),
triangle blocks (32 rows) and tiles (128 x 64)."""
import ctypes

import numpy as np
import pytest

from rigidfibers_kth_b200 import _lib as L

pytestmark = pytest.mark.gpu


def dgesv(A, b):
    n = len(b)
    x, piv, info = np.zeros(n), np.zeros(n, dtype=np.int32), ctypes.c_int32(-1)
    dp = ctypes.POINTER(ctypes.c_double)
    L.check(L.lib().rf_dgesv(n, A.ctypes.data_as(dp), n, b.ctypes.data_as(dp), x.ctypes.data_as(dp), piv.ctypes.data,
                             ctypes.byref(info), 0))
    return x, piv, info.value


def check(A, b, x, piv):
    """Pivots equal LAPACK's order as torch's LU finds it on the same matrix
    (continuous random entries: no ties), and the backward error
    |b - A x| / (|A| |x|) is within n units of rounding."""
    import torch

    At = torch.from_numpy(np.ascontiguousarray(A)).cuda()
    _, ref = torch.linalg.lu_factor(At)
    assert np.array_equal(piv, ref.cpu().numpy())
    xt, bt = torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda()
    r = (bt - At @ xt).norm() / (At.norm() * xt.norm())
    assert float(r) <= len(b) * 2.0 ** -53


@pytest.mark.parametrize("n", [2, 31, 32, 33, 96, 127, 128, 129, 160, 161, 193, 255, 256, 257, 385, 1000])
def test_random_matrices(n):
    rng = np.random.default_rng(n)
    A, b = np.asfortranarray(rng.standard_normal((n, n))), rng.standard_normal(n)
    x, piv, info = dgesv(A, b)
    assert info == 0
    check(A, b, x, piv)


# a few rows over 4096, 8192 and 16384: the first sub-panels are of each width
@pytest.mark.parametrize("n", [4100, 8200, 16390])
def test_register_sub_panels(n):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64).cpu().numpy().T  # column-major
    b = np.random.default_rng(n).standard_normal(n)
    x, piv, info = dgesv(A, b)
    assert info == 0
    check(A, b, x, piv)


def test_repeated_rows_ties_and_singular():
    """Every row's largest entry tied in magnitude with others': the first row of
    largest magnitude is the pivot (idamax); a repeated pivot row far below the
    panel; a zero column deep in a later panel reports LAPACK's info."""
    n = 300
    rng = np.random.default_rng(5)
    A = np.asfortranarray(rng.choice([-1.0, 1.0], size=(n, n)) + 0.0)
    A[np.arange(n), np.arange(n)] *= 1.0
    b = rng.standard_normal(n)
    import scipy.linalg as sl

    x, piv, info = dgesv(A, b)
    lu, ref = sl.lu_factor(A)
    # exact arithmetic of small integers until the first rounding: the leading
    # pivots are decided by ties alone
    assert info == 0
    assert np.array_equal(piv[:3], ref[:3] + 1)
    assert np.linalg.norm(A @ x - b) <= 1e-10 * np.linalg.norm(b) * np.linalg.cond(A)
    Z = np.asfortranarray(rng.standard_normal((n, n)))
    Z[:, 200] = 0.0
    _, _, info = dgesv(Z, b)
    assert info == 201
