"""The FP64 blocks of distant pairs are no further from extended precision than
the reference's own formulas in FP64 (the oracle), at every start of the
backward recursion: assembled blocks and the matrix-free product."""
import numpy as np
import pytest

import rigidfibers_kth_b200 as rf
from oracle import rfo

pytestmark = pytest.mark.gpu
LD = np.longdouble


def moments(R, t, N):
    """I_n, J_n, S_n (Int_analytical.f90:96-207) by the backward recursion from
    n = 90, in 64-bit mantissas: for |R| >= 3 truncation is below 1e-30."""
    b, c = -2 * (R @ t), (R * R).sum(-1)
    ue, ub = np.sqrt(1 + b + c), np.sqrt(1 - b + c)
    z = np.zeros_like(c)
    i1, i2, j1, j2, s1, s2 = z, z, z, z, z, z
    out = []
    for n in range(90, -1, -1):
        w = 2 * b / (ue + ub) if n % 2 else ue + ub
        i0 = (w - (n + LD(1.5)) * b * i1 - (n + 2) * i2) / ((n + 1) * c)
        j0 = (i0 - b * j1 - j2) / c
        s0 = (j0 - b * s1 - s2) / c
        i1, i2, j1, j2, s1, s2 = i0, i1, j0, j1, s0, s1
        if n < N + 3:
            out.append((i0, j0, s0))
    return [np.stack(v, -1) for v in zip(*out[::-1])]


def block(x, t, xs, ts, N, NoQI, eps):
    """The 3N x 3N block of target (x, t) and source (xs, ts) (matrix_assembly.f90:407-629)."""
    g, h = np.sqrt(LD(3) / 5), LD(1) / NoQI
    s = np.array([-1 + (2 * i + 1 + z) * h for i in range(NoQI) for z in (-g, LD(0), g)])
    w = np.array([v * h / 9 for _ in range(NoQI) for v in (LD(5), LD(8), LD(5))])
    leg = np.zeros((N + 1, N + 3), dtype=LD)  # P_m from P_m-1, P_m-2
    leg[0, 0], leg[1, 1] = 1, 1
    for m in range(2, N + 1):
        leg[m, 1:] = LD(2 * m - 1) * leg[m - 1, :-1]
        leg[m] = (leg[m] - (m - 1) * leg[m - 2]) / m
    P = (leg[:, :N + 1] @ (s ** np.arange(N + 1)[:, None])).astype(LD)
    R = (x - xs) + s[:, None] * t
    I, J, S = moments(R, ts, N)
    e = 2 * LD(eps) ** 2
    L = lambda a, k: a[:, k:k + N + 1] @ leg[:, :N + 1].T  # noqa: E731
    u = lambda v: v[..., None, None]  # noqa: E731
    RR, pR = R[:, None, :, None] * R[:, None, None, :], ts[:, None] * R[:, None, None, :]
    G = (u(L(I, 0) + e * L(J, 0)) * np.eye(3, dtype=LD) + u(L(J, 0) - 3 * e * L(S, 0)) * RR
         + u(-L(J, 1) + 3 * e * L(S, 1)) * (pR + pR.swapaxes(-1, -2))
         + u(L(J, 2) - 3 * e * L(S, 2)) * (ts[:, None] * ts[None, :]))
    th = np.einsum("kq,qmab->kmab", w * P, G)
    d = -np.log(LD(eps) ** 2 * np.exp(LD(1)))
    lam = np.concatenate([[LD(0)], np.cumsum([LD(2) / k for k in range(1, N + 1)])])
    B = np.zeros((3 * N, 3 * N), dtype=LD)
    for k in range(1, N + 1):
        tt = t[:, None] * np.einsum("a,mab->mb", t, th[k])[:, None, :]
        v = (LD(0.75) / (d - 2) * tt if k == 1 else
             LD(0.5) * (2 * k + 1) / (d + 2 - lam[k]) * (th[k] - (d - 2 - lam[k]) / 2 / (d - lam[k]) * tt))
        B[3 * k - 3:3 * k] = v[1:].transpose(1, 0, 2).reshape(3, 3 * N)
    return B


# squared centre distances that put target points just above and below every
# start of the recursion (c = 16, 45, 65, 105, 190, 420) and far beyond
@pytest.mark.parametrize("c", [20.0, 30.0, 38.0, 48.0, 60.0, 75.0, 95.0, 130.0, 210.0, 280.0, 440.0, 1000.0])
@pytest.mark.parametrize("N", [5, 8])
def test_error_against_the_reference_formulas(N, c):
    rng = np.random.default_rng(int(c) + N)
    M, eps = 64, 1e-2
    d = rng.normal(size=(M, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    ori = rng.normal(size=(M, 3))
    ori /= np.linalg.norm(ori, axis=1, keepdims=True)
    pos = np.sqrt(c) * d
    pos[0] = 0.0  # the source; the others are its targets
    x = np.zeros(3 * N * M)
    x[:3 * N] = rng.normal(size=3 * N)
    p = rf.FiberParams(slenderness=eps, num_terms_in_force_expansion=N)
    with rf.Simulation(rf.Configuration(p, pos, ori)) as s:
        s.assemble_system()
        A, y = s.matrix(), s.matvec_free(x)
    A_o, _ = rfo.assemble_system(rfo.make_params(M, N=N, eps=eps), pos, ori)
    blocks, products = [], []
    for i in range(1, M):
        r = slice(3 * N * i, 3 * N * (i + 1))
        B = block(pos[i].astype(LD), ori[i].astype(LD), pos[0].astype(LD), ori[0].astype(LD), N, 8, eps)
        yb = B @ x[:3 * N]
        # per weight l of the source's expansion, relative to the block
        blocks.append([(np.abs(a[r, :3 * N] - B) / np.abs(B).max()).reshape(3 * N, N, 3).max((0, 2)) for a in (A, A_o)])
        products.append([np.abs(v - yb).max() / np.abs(yb).max() for v in (y[r], A_o[r, :3 * N] @ x[:3 * N])])
    # Mean and median over 63 directions (the mean is ruled by the few near the
    # source's axis, where both follow the same closed forms).  The entries are
    # mixed differences of G, 1 / c of its size, so that a rounding of geometry,
    # moments or projections, which both have, is c units: four of them.
    for stat in (np.mean, np.median):
        if N <= 5:  # the assembly's recursion; above, its closed forms are the reference's
            m = stat(np.array(blocks, dtype=float), 0)
            assert (m[0] <= m[1] + 4 * c * 2.0 ** -52).all(), m
        m = stat(np.array(products, dtype=float), 0)
        assert m[0] <= m[1] + 4 * c * 2.0 ** -52, m
