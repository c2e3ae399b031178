"""Products with few and many column splits: the partial sums' reduction at
sizes around its groups of 64 (FP64) and 128 (FP32) rows, odd sizes, and from
one split to hundreds, against numpy on the stored matrix."""
import numpy as np
import pytest

import rigidfibers_kth_b200 as rf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(1, 1), (2, 5), (9, 5), (43, 1), (43, 5), (86, 1), (127, 4), (128, 3), (301, 5)])
@pytest.mark.parametrize("precision", [rf.PREC_FP64, rf.PREC_FP32, rf.PREC_MIXED_BF16])
def test_product(M, N, precision):
    """Sums of n products in the accumulator's precision: n units of it (half,
    for rounding to nearest) relative to |A| |x|."""
    pos, ori = rf.generate_layout(M, "uniform", (M / 8.0) ** (1 / 3) + 0.5, 0.2, seed=M)
    p = rf.FiberParams(slenderness=1e-2, num_terms_in_force_expansion=N, precision=precision)
    with rf.Simulation(rf.Configuration(p, pos, ori)) as s:
        s.assemble_system()
        A = s.matrix_rows(0, s.n, inner=True)  # what matvec multiplies by: the BF16 matrix where there is one
        x = np.random.default_rng(N).normal(size=s.n)
        y = s.matvec(x)
    unit = 2.0 ** -24 if precision == rf.PREC_FP32 else 2.0 ** -53
    assert np.all(np.abs(y - A @ x) <= (len(x) + 4) * unit * (np.abs(A) @ np.abs(x)))
