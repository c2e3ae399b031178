"""The device-controlled GMRES (restart lengths up to 16) against the oracle's
solver on the same matrix: iterates, iteration counts, budget, cold and warm
starts, and the host-controlled solver above that length."""
import numpy as np
import pytest

import rigidfibers_kth_b200 as rf
from oracle import rfo

pytestmark = pytest.mark.gpu


def system(M, **kw):
    pos, ori = rf.generate_layout(M, "uniform", (M / 8.0) ** (1 / 3), 0.2, seed=40 + M)
    sim = rf.Simulation(rf.Configuration(rf.FiberParams(slenderness=1e-3, **kw), pos, ori))
    sim.assemble_system()
    return sim, np.array(sim.matrix(), order="F"), sim.rhs()


# restart 1 (every cycle one step), the reference's 10, the last
# device-controlled length and the first host-controlled one; 3 iterations
# end inside a cycle, on its last step and before convergence
@pytest.mark.parametrize("restart,tol,budget", [(1, 1e-4, 400), (3, 1e-8, 3), (10, 1e-10, 300), (10, 1e-13, 300),
                                                (16, 1e-10, 16), (16, 1e-12, 300), (17, 1e-12, 300)])
@pytest.mark.parametrize("M", [1, 2, 37])
def test_iterates_match_oracle(M, restart, tol, budget):
    sim, A, b = system(M, gmres_restart=restart, gmres_tol=tol, gmres_max_iters=budget)
    with sim:
        sim.solve_system()
        x, st = sim.coeffs(), sim.solve_stats()
    x_o, info, iters, be = rfo.solve_gmres(A, b, restart=restart, max_iters=budget, tol=tol)
    assert st["converged"] == (info == 0)
    # both end on a residual within a few units of rounding of each other; the
    # count may move by one where the estimate meets 1e-13 at that level
    assert abs(st["iterations"] - iters) <= (1 if tol < 1e-12 else 0)
    assert np.abs(x - x_o).max() <= 1e-10 * max(1e-30, np.abs(x_o).max())


@pytest.mark.parametrize("precision,tol", [(rf.PREC_FP64, 1e-10), (rf.PREC_FP32, 1e-5)])
def test_warm_start_zero_rhs_and_true_residual(precision, tol):
    """A start from the solution ends at once; the residual reported is the
    true one; without external force b = 0 and x = 0 whatever the start."""
    sim, A, b = system(37, gmres_tol=tol, gmres_max_iters=300, precision=precision)
    with sim:
        assert sim.solve_system() == 0
        x, st = sim.coeffs(), sim.solve_stats()
        true = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
        # the device forms the residual from sums of n = 555 products in the
        # storage precision: n * eps of |A| |x| ~ 3 |b| on top
        eps = 2.0 ** -53 if precision == rf.PREC_FP64 else 2.0 ** -24
        assert st["residual"] <= tol and abs(st["residual"] - true) <= 3 * 555 * eps
        its = st["iterations"]
        assert sim.solve_system() == 0  # from x
        assert sim.solve_stats()["iterations"] <= 2 < its
    sim, A, b = system(5, gmres_tol=tol, precision=precision, external_force=(0.0, 0.0, 0.0))
    with sim:
        z = np.zeros(15)
        sim.set_history(z, z + 1.0, z, z, np.ones(75))
        assert np.abs(b).max() == 0.0
        assert sim.solve_system() == 0
        assert np.abs(sim.coeffs()).max() == 0.0


# one CTA's rows and the next (148 rows a fiber pair more or less), ragged
# 64-row tiles, the largest system of the single-kernel solver and the first
# beyond it (N = 4: 12 rows a fiber, 8184 and 8196); the product timer takes the
# kernel-per-pass solver on the same system
@pytest.mark.parametrize("M,N,restart", [(9, 5, 10), (10, 5, 10), (43, 1, 7), (50, 3, 16), (682, 4, 10), (683, 4, 10)])
def test_single_kernel_solver_matches_launched_passes(M, N, restart):
    pos, ori = rf.generate_layout(M, "gaussian", 3.0 * (M / 1000.0) ** (1 / 3), 0.2, seed=M)
    p = rf.FiberParams(slenderness=1e-3, num_terms_in_force_expansion=N, gmres_restart=restart, gmres_tol=1e-11,
                       gmres_max_iters=300)
    with rf.Simulation(rf.Configuration(p, pos, ori)) as sim:
        sim.assemble_system()
        out = []
        for timed in (False, True):
            sim.set_history(pos, ori, pos, ori, np.zeros(3 * N * M))
            sim.gemv_timer(timed)
            assert sim.solve_system() == 0
            out.append((sim.coeffs(), sim.solve_stats()))
    (x, a), (y, b) = out
    assert a["iterations"] == b["iterations"] and a["matvecs"] == b["matvecs"]
    # the same steps; sums of n products and n squares in another order: a few n
    # units of rounding of |x|, far below 1e-11
    assert np.abs(x - y).max() <= 1e-11 * np.abs(y).max()


def test_one_rank_communicator_above_the_single_kernel_solver():
    """A system too large for the single-kernel solver: every product of a
    one-rank sharded handle goes through the all-gather and the compaction, and
    steps exactly like the whole system's."""
    M = 560
    pos, ori = rf.generate_layout(M, "gaussian", 2.0, 0.2, seed=2103)
    out = []
    for sharded in (False, True):
        kw = dict(nccl_id=rf.shard_unique_id()) if sharded else {}
        p = rf.FiberParams(slenderness=1e-3, gmres_tol=1e-10, gmres_max_iters=300, shard_index=0, shard_count=1)
        with rf.Simulation(rf.Configuration(p, pos, ori), **kw) as s:
            for t in range(2):
                assert s.step(t) == 0
            out.append(s.state() + s.velocities() + (s.coeffs(), s.rhs()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("restart", [1, 2, 5, 10, 16])
@pytest.mark.parametrize("passes", [False, True])
def test_restarts_without_a_product(restart, passes):
    """The residual of a restart comes from the cycle's basis: the iterates stay
    the oracle's, which makes the product, over many short cycles, in the
    single-kernel solver and in launched passes; products are made for the start
    and for the accepted solution only."""
    sim, A, b = system(37, gmres_restart=restart, gmres_tol=1e-10, gmres_max_iters=600)
    with sim:
        sim.gemv_timer(passes)
        assert sim.solve_system() == 0
        x, st = sim.coeffs(), sim.solve_stats()
    x_o, info, iters, _ = rfo.solve_gmres(A, b, restart=restart, max_iters=600, tol=1e-10)
    assert info == 0 and st["iterations"] == iters and iters > restart
    assert st["matvecs"] == iters + 2
    assert np.linalg.norm(b - A @ x) <= 1e-10 * np.linalg.norm(b) * (1 + 1e-4)
    assert np.abs(x - x_o).max() <= 1e-10 * np.abs(x_o).max()


# rows per CTA of the single-kernel solver that are not whole groups of eight,
# with four, two and one columns in flight per warp, even and odd sizes (M = 1: b = 0)
@pytest.mark.parametrize("M,N,restart", [(1, 5, 10), (2, 5, 10), (101, 5, 10), (193, 5, 16), (333, 3, 5), (345, 5, 10)])
def test_single_kernel_solver_row_shapes(M, N, restart):
    sim, A, b = system(M, num_terms_in_force_expansion=N, gmres_restart=restart, gmres_tol=1e-12, gmres_max_iters=300)
    with sim:
        assert sim.solve_system() == 0
        x, st = sim.coeffs(), sim.solve_stats()
    # the true residual was accepted; numpy's differs by the rounding of n products
    r, norm = np.linalg.norm(b - A @ x), np.linalg.norm(b)
    assert r <= (1e-12 + 3 * len(b) * 2.0 ** -53) * norm
    assert abs(st["residual"] * norm - r) <= 3 * len(b) * 2.0 ** -53 * norm


def test_past_breakdown():
    """Six unknowns, a tolerance that is never met: the Krylov space is exhausted
    after six steps at most, where the next vector is rounding and its norm is
    not |w|^2 - |h2|^2; six more steps on what that leaves keep the solution (n
    units of rounding times a condition below 100)."""
    sim, A, b = system(2, num_terms_in_force_expansion=1, gmres_restart=16, gmres_tol=1e-18, gmres_max_iters=12)
    with sim:
        sim.solve_system()
        x = sim.coeffs()
    assert np.linalg.cond(A) < 100
    x_o = np.linalg.solve(A, b)
    assert np.abs(x - x_o).max() <= 1e-13 * np.abs(x_o).max()
