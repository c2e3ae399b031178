"""Rounding of the pair sums with the numeric integral: each source's points are
summed by themselves before the sources are."""
import numpy as np
import pytest

import rigidfibers_kth_b200 as rf

pytestmark = pytest.mark.gpu
LD = np.longdouble


def velocity_integral(x, t, pos, ori, coeffs, eps):
    """IF_0 of one target over sources with the force F / 2 + a s (N = 1, eight
    intervals), in 64-bit mantissas."""
    g, h = np.sqrt(LD(3) / 5), LD(1) / 8
    s = np.array([-1 + (2 * i + 1 + z) * h for i in range(8) for z in (-g, LD(0), g)])
    w = np.array([v * h / 9 for _ in range(8) for v in (LD(5), LD(8), LD(5))])
    R = (x + s[:, None] * t)[:, None, None] - (pos[:, None] + s[:, None] * ori[:, None])[None]  # q, j, s
    r = np.sqrt((R * R).sum(-1))
    e = 2 * LD(eps) ** 2
    f = np.array([0, 0, LD(-0.5)]) + s[:, None] * coeffs[:, None, :]  # j, s
    Rf = np.einsum("qjsa,jsa->qjs", R, f)
    u = (1 / r + e / r ** 3)[..., None] * f + ((1 / r ** 3 - 3 * e / r ** 5) * Rf)[..., None] * R
    return np.einsum("q,s,qjsa->a", w, w, u)


def test_small_sources_after_a_large_one():
    """The first source's velocity is B, every other one's about three units in the
    last place of B (2000 sources: 55 to a chunk).  Added source by source, the
    first chunk's others round to whole units: a random walk of 54 halves, 2 units
    rms, and a few units of the large source's own.  Point by point, 24 terms of an
    eighth of a unit each, all would be lost: 160 units.  The line lies at 30."""
    M, eps = 2000, 1e-2
    rng = np.random.default_rng(1)
    pos = rng.uniform(-2, 2, (M, 3)) + [20.0, 0.0, 0.0]
    ori = rng.normal(size=(M, 3))
    ori /= np.linalg.norm(ori, axis=1, keepdims=True)
    pos[0], ori[0] = [3.0, 0.0, 0.0], [1.0, 0.0, 0.0]
    pos[-1], ori[-1] = 0.0, [0.0, 1.0, 0.0]  # the target
    a = np.zeros((M, 3))
    o = slice(1, M - 1)
    args = [v.astype(LD) for v in (pos, ori)]
    small = velocity_integral(args[0][-1], args[1][-1], args[0][o], args[1][o], a[o].astype(LD), eps)[2] / (M - 2)
    first = lambda v: velocity_integral(args[0][-1], args[1][-1], args[0][:1], args[1][:1], v, eps)[2]  # noqa: E731
    one = first(np.array([[0, 0, LD(1)]])) - first(np.zeros((1, 3), dtype=LD))
    a[0, 2] = float(small / one * 2.0 ** 53 / 6)  # B = small / 3 units, a unit between 2^-53 and 2^-52 of B
    p = rf.FiberParams(slenderness=eps, use_analytical_integration=0, num_terms_in_force_expansion=1,
                       precision=rf.PREC_FP32)
    z = np.zeros(3 * M)
    with rf.Simulation(rf.Configuration(p, pos, ori)) as sim:
        sim.set_history(pos, ori, z, z, a.reshape(-1))
        sim.set_state(pos, ori)
        sim.update_velocities()
        V = sim.velocities()[0].reshape(M, 3)[-1]
    IF = velocity_integral(args[0][-1], args[1][-1], args[0][:-1], args[1][:-1], a[:-1].astype(LD), eps)[2]
    d = -np.log(LD(eps) ** 2 * np.exp(LD(1)))
    err = float(V[2] * 2 * d + (d + 2) - IF)  # V_z = (-(d + 2) / 2 + IF / 2) / d across the force
    unit = np.spacing(abs(float(IF)))
    print("error %.1f units; the others add %.1f" % (err / unit, float(small) * (M - 2) / unit))
    assert abs(err) <= 30 * unit
