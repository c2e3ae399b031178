"""Pivots of the device LU where many rows tie: A = P L U of small integers and
halves, so that every step is exact and idamax's first maximum decides alone."""
import ctypes

import numpy as np
import pytest

from rigidfibers_kth_b200 import _lib as L

pytestmark = pytest.mark.gpu


def tied_matrix(n, seed):
    """L's rows by the row of A they belong to, U, and the pivot positions.

    Step k's pivot stands at position piv[k] of the rows as the earlier swaps left
    them: rows between k and there have multipliers of at most a half, a third of
    those beyond tie with it.  Pivots come from the warp of the diagonal, from its
    CTA (256 rows), from far CTAs, and from one far position ten times running."""
    rng = np.random.default_rng(seed)
    rows = np.arange(n)
    Lr = np.zeros((n, n))
    piv = np.zeros(n, dtype=np.int64)
    far = n - 1 - n // 7
    for k in range(n):
        if k % 50 < 10 and k <= far:
            p = far
        else:
            p = min(n - 1, k + int(rng.choice([0, 1, rng.integers(0, 32), rng.integers(0, 256), rng.integers(0, n)])))
        l = rng.choice([-0.5, 0.0, 0.0, 0.5], n - k)
        l[p - k] = 1.0
        tail = l[p - k + 1:]
        tie = rng.random(len(tail)) < 1 / 3
        tail[tie] = rng.choice([-1.0, 1.0], tie.sum())
        Lr[rows[k:], k] = l
        rows[k], rows[p] = rows[p], rows[k]
        piv[k] = p
    U = np.triu(rng.choice([-1.0, 0.0, 0.0, 1.0], (n, n)), 1)
    U[np.arange(n), np.arange(n)] = rng.choice([-4.0, -2.0, -1.0, 1.0, 2.0, 4.0], n)
    return Lr, U, piv


# 4200 and 8300: sub-panels of two and four rows a thread (16 CTAs)
@pytest.mark.parametrize("n", [40, 300, 1000, 4200, 8300])
def test_first_maximum_everywhere(n):
    import torch

    Lr, U, piv = tied_matrix(n, n)
    # exact: multiples of a half below 2^17
    A = (torch.from_numpy(Lr).cuda() @ torch.from_numpy(U).cuda()).cpu().numpy()
    x0 = np.random.default_rng(1).integers(-8, 9, n).astype(np.float64)
    b = A @ x0
    A = np.asfortranarray(A)
    x, got, info = np.zeros(n), np.zeros(n, dtype=np.int32), ctypes.c_int32(-1)
    dp = ctypes.POINTER(ctypes.c_double)
    L.check(L.lib().rf_dgesv(n, A.ctypes.data_as(dp), n, b.ctypes.data_as(dp), x.ctypes.data_as(dp), got.ctypes.data,
                             ctypes.byref(info), 0))
    assert info.value == 0
    assert np.array_equal(got, piv + 1)
    assert np.array_equal(x, x0)  # every intermediate value is a small multiple of a half
