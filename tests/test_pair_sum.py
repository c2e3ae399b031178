"""The pair sums (recomputed velocities, matrix-free product) against the
oracle at the edges of their batches, chunks, target groups and block sizes."""
import numpy as np
import pytest

import rigidfibers_kth_b200 as rf
from oracle import rfo

pytestmark = pytest.mark.gpu


# one fiber, a last batch of one source (17, 33), more targets than a CTA's
# four, several chunks (150); 3 to 48 points; N past the split of the moment
# recursion's tail (5 | 6) and the largest
@pytest.mark.parametrize("M,N,NoQI", [(1, 5, 8), (2, 5, 1), (17, 5, 8), (33, 1, 16), (33, 8, 9), (34, 6, 8), (19, 7, 3),
                                      (150, 5, 8), (150, 4, 5)])
@pytest.mark.parametrize("analytic", [1, 0])
def test_against_oracle(M, N, NoQI, analytic):
    rng = np.random.default_rng(1000 * M + 10 * N + NoQI)
    side = int(np.ceil(M ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3), -1).reshape(-1, 3)[:M]
    pos = 2.2 * grid + rng.uniform(-0.4, 0.4, (M, 3))
    ori = rng.normal(size=(M, 3))
    ori /= np.linalg.norm(ori, axis=1, keepdims=True)
    x = rng.normal(size=3 * N * M)
    p = rf.FiberParams(slenderness=1e-2, num_terms_in_force_expansion=N, num_quadrature_intervals=NoQI,
                       use_analytical_integration=analytic)
    z = np.zeros(3 * M)
    with rf.Simulation(rf.Configuration(p, pos, ori)) as s:
        s.set_history(pos, ori, z, z, x)
        s.set_state(pos, ori)
        y = s.matvec_free(x)
        s.update_velocities()
        V, W = s.velocities()
    po = rfo.make_params(M, N=N, NoQI=NoQI, eps=1e-2, analytic=bool(analytic))
    A, _ = rfo.assemble_system(po, pos, ori)
    V_o, W_o = rfo.velocities(po, pos, ori, x)
    # the FP64 contract, or three times what one unit in the last place of the
    # positions moves where fibers pass close to one another
    pp = pos * (1 + 2.0 ** -52)
    Ap, _ = rfo.assemble_system(po, pp, ori)
    V_p, W_p = rfo.velocities(po, pp, ori, x)
    for got, ref, moved in ((y, A @ x, Ap @ x), (V, V_o, V_p), (W, W_o, W_p)):
        scale = max(np.abs(ref).max(), np.abs(V_o).max())
        tol = max(1e-10, 3 * np.abs(moved - ref).max() / scale)
        assert np.isfinite(got).all()
        assert np.abs(got - ref).max() <= tol * scale
