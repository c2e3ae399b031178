"""The FP64 analytic assembly's edges against the oracle: point distances on
both sides of every line of the moment recursion (c = 10 and the starts of the
backward recursion), the cone about the source axis, ragged target groups,
quadrature sizes on both sides of its tiles, velocity panels."""
import numpy as np
import pytest

import rigidfibers_kth_b200 as rf
from oracle import rfo

pytestmark = pytest.mark.gpu


def assembled(pos, ori, eps, N, NoQI, reuse=0):
    p = rf.FiberParams(slenderness=eps, num_terms_in_force_expansion=N, num_quadrature_intervals=NoQI,
                       velocity_mode=reuse, gmres_tol=1e-13, gmres_max_iters=1000)
    with rf.Simulation(rf.Configuration(p, pos, ori)) as s:
        s.assemble_system()
        A, b = s.matrix(), s.rhs()
        s.solve_system()
        s.update_velocities()
        return A, b, s.coeffs(), s.velocities()


def unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


# squared centre distances so that the target points straddle c = 10, 13, 16,
# 20, 30, 48, 80, 150, and one and four decades beyond
@pytest.mark.parametrize("c", [9.0, 10.5, 13.0, 16.0, 20.0, 30.0, 48.0, 80.0, 150.0, 1e3, 1e6])
@pytest.mark.parametrize("eps", [1e-3, 1e-2])
def test_distances(c, eps):
    """Five fibers around a sixth at the same distance, in directions from
    across its axis to 4 degrees off it.  Norm-wise 1e-10, the FP64 contract."""
    rng = np.random.default_rng(int(c))
    ang = np.radians([90.0, 60.0, 35.0, 12.0, 4.0])
    p = np.array([0.0, 0.0, 1.0])
    d = np.stack([np.sin(ang) * np.cos(7 * ang), np.sin(ang) * np.sin(7 * ang), np.cos(ang)], 1)
    pos = np.concatenate([[[0.0, 0.0, 0.0]], np.sqrt(c) * d])
    ori = np.concatenate([[p], unit(rng.normal(size=(5, 3)))])
    A, b, _, _ = assembled(pos, ori, eps, 5, 8)
    A_o, b_o = rfo.assemble_system(rfo.make_params(6, eps=eps), pos, ori)
    assert np.abs(A - A_o).max() <= 1e-10 * np.abs(A_o).max()
    assert np.abs(b - b_o).max() <= 1e-10 * np.abs(b_o).max()


@pytest.mark.parametrize("M,N,NoQI", [(1, 5, 8), (2, 1, 1), (3, 2, 2), (4, 3, 4), (5, 4, 5), (15, 5, 7), (16, 5, 8),
                                      (17, 5, 9), (33, 5, 16), (21, 1, 16), (18, 3, 11)])
@pytest.mark.parametrize("reuse", [0, 1])
def test_ragged_sizes(M, N, NoQI, reuse):
    rng = np.random.default_rng(100 * M + N)
    side = int(np.ceil(M ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3), -1).reshape(-1, 3)[:M]
    pos = 1.7 * grid + rng.uniform(-0.3, 0.3, (M, 3))
    ori = unit(rng.normal(size=(M, 3)))
    A, b, x, (V, W) = assembled(pos, ori, 1e-2, N, NoQI, reuse)
    p = rfo.make_params(M, N=N, NoQI=NoQI, eps=1e-2)
    A_o, b_o = rfo.assemble_system(p, pos, ori)
    # 1e-10, or three times what one unit in the last place of the positions moves
    A_p, _ = rfo.assemble_system(p, pos * (1 + 2.0 ** -52), ori)
    tol = max(1e-10, 3 * np.abs(A_p - A_o).max() / np.abs(A_o).max())
    assert np.abs(A - A_o).max() <= tol * np.abs(A_o).max()
    assert np.abs(b - b_o).max() <= tol * max(1e-30, np.abs(b_o).max())
    V_o, W_o = rfo.velocities(p, pos, ori, x)
    assert np.abs(V - V_o).max() <= 1e-10 * np.abs(V_o).max()
    assert np.abs(W - W_o).max() <= 1e-10 * max(np.abs(W_o).max(), np.abs(V_o).max())


@pytest.mark.parametrize("N,NoQI", [(1, 3), (3, 8), (5, 8), (8, 8)])
@pytest.mark.parametrize("gap", [0.3, 0.05, 0.01])
@pytest.mark.parametrize("eps", [1e-3, 1e-2])
def test_numeric_integral_of_close_pairs(N, NoQI, gap, eps):
    """The numeric inner integral of two crossing fibers.  Both sides round the
    positions (a few units of |x| <= 2, relative to the gap) under a fifth power
    of the distance: 5 x 2 units, four times for the sums."""
    rng = np.random.default_rng(int(1000 * gap) + N)
    t = unit(rng.normal(size=(2, 3)))
    s = rng.uniform(-0.9, 0.9, 2)
    pos = np.array([[0.0, 0.0, 0.0], gap * unit(np.cross(t[0], t[1])) + s[0] * t[0] - s[1] * t[1]])
    p = rf.FiberParams(slenderness=eps, num_terms_in_force_expansion=N, num_quadrature_intervals=NoQI,
                       use_analytical_integration=0)
    with rf.Simulation(rf.Configuration(p, pos, t)) as sim:
        sim.assemble_system()
        A, b = sim.matrix(), sim.rhs()
    A_o, b_o = rfo.assemble_system(rfo.make_params(2, N=N, NoQI=NoQI, eps=eps, analytic=False), pos, t)
    tol = 40 * 2.0 ** -52 * (1 + 2 / gap)
    assert np.abs(A - A_o).max() <= tol * np.abs(A_o).max()
    assert np.abs(b - b_o).max() <= tol * np.abs(b_o).max()
