"""FP64 analytic fibers so far apart that the powers of the distance leave the
FP64 range (c^2.5 from 1e61 half-lengths on): each is isolated, and nothing in
the system may be non-finite."""
import numpy as np
import pytest

import rigidfibers_kth_b200 as rf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [5, 7])
@pytest.mark.parametrize("scale", [1e45, 1e52, 1e61, 1e63, 1e80, 1e120])
def test_isolated_fibers(N, scale):
    """A = I and y = x within 1e-10, the FP64 contract, and an isolated fiber's
    velocity (coeffs_and_vels.f90:698-705)."""
    rng = np.random.default_rng(N)
    M, eps = 8, 1e-3
    pos = scale * rng.normal(size=(M, 3))
    ori = rng.normal(size=(M, 3))
    ori /= np.linalg.norm(ori, axis=1, keepdims=True)
    p = rf.FiberParams(slenderness=eps, num_terms_in_force_expansion=N, gmres_tol=1e-10)
    with rf.Simulation(rf.Configuration(p, pos, ori)) as s:
        s.assemble_system()
        assert np.abs(s.matrix() - np.eye(s.n)).max() <= 1e-10
        x = rng.normal(size=s.n)
        assert np.abs(s.matvec_free(x) - x).max() <= 1e-10
        assert s.solve_system() == 0
        s.update_velocities()
        V, W = s.velocities()
    d = -np.log(eps * eps * np.e)
    F = np.array([0.0, 0.0, -1.0])
    Vi = 0.5 * ((d + 2.0) * F + (d - 2.0) * (ori @ F)[:, None] * ori) / d
    assert np.abs(V.reshape(M, 3) - Vi).max() <= 1e-10
    assert np.abs(W).max() <= 1e-10
