"""Solves without a right-hand side (one fiber, or no external force): x = 0
whatever the start holds, and no product is made."""
import numpy as np
import pytest

import rigidfibers_kth_b200 as rf

pytestmark = pytest.mark.gpu


# the single-kernel solver, launched passes (the product timer on; above its
# size; FP32) and the host-controlled solver (restart 17)
@pytest.mark.parametrize("M,restart,precision,timed", [
    (1, 10, rf.PREC_FP64, False), (9, 10, rf.PREC_FP64, False), (9, 10, rf.PREC_FP64, True),
    (9, 17, rf.PREC_FP64, True), (560, 10, rf.PREC_FP64, False), (9, 10, rf.PREC_FP32, True)])
@pytest.mark.parametrize("start", [0.0, 1.0, np.nan, np.inf])
def test_zero_rhs(M, restart, precision, timed, start):
    pos, ori = rf.generate_layout(M, "uniform", (M / 8.0) ** (1 / 3), 0.2, seed=3)
    p = rf.FiberParams(slenderness=1e-3, gmres_restart=restart, gmres_tol=1e-6, precision=precision,
                       external_force=(0.0, 0.0, 0.0) if M > 1 else (0.0, 0.0, -1.0))
    with rf.Simulation(rf.Configuration(p, pos, ori)) as s:
        z = np.zeros(3 * M)
        s.set_history(z, z + 1.0, z, z, np.full(s.n, start))
        s.assemble_system()
        assert np.abs(s.rhs()).max() == 0.0
        s.gemv_timer(timed)
        assert s.solve_system() == 0
        assert np.array_equal(s.coeffs(), np.zeros(s.n))
        st = s.solve_stats()
        assert st["converged"] and st["iterations"] == 0 and st["matvecs"] == 0
        if timed:
            assert s.gemv_timer(False)[0] == 0
