"""The FP64-integrated pairs of the split (mixed-precision) assembly against the
oracle: every pair near (a threshold beyond all distances), so that each group
size of a warp, quadrature size and distance goes through the near-pair kernel,
with and without its block buffer."""
import numpy as np
import pytest
import torch

import rigidfibers_kth_b200 as rf
from oracle import rfo

pytestmark = pytest.mark.gpu


def suspension(M, seed):
    rng = np.random.default_rng(seed)
    side = int(np.ceil(M ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3), -1).reshape(-1, 3)[:M]
    ori = rng.normal(size=(M, 3))
    return 1.7 * grid + rng.uniform(-0.3, 0.3, (M, 3)), ori / np.linalg.norm(ori, axis=1, keepdims=True)


def params(N, NoQI, precision=rf.PREC_MIXED_BF16, **kw):
    return rf.FiberParams(slenderness=1e-2, num_terms_in_force_expansion=N, num_quadrature_intervals=NoQI,
                          precision=precision, near_field_c=1e6, **kw)


@pytest.mark.parametrize("M,N,NoQI", [(2, 5, 8), (4, 5, 8), (5, 5, 8), (6, 5, 7), (17, 5, 8), (18, 5, 9), (33, 5, 16),
                                      (9, 1, 1), (10, 2, 2), (19, 3, 5), (23, 4, 11)])
@pytest.mark.parametrize("reuse", [0, 1])
def test_all_pairs_near(M, N, NoQI, reuse):
    """Entries: FP64 integrals rounded to FP32 (2^-24 of the entry; 2^-23 leaves
    room for the integrals' own error), which themselves agree to 1e-9 of the
    largest entry, or three times what one unit in the last place of the
    positions moves.  Right-hand side: FP64.  Velocities: 3 N M products of FP32
    panel entries, each off by 2^-24 of itself."""
    pos, ori = suspension(M, M + 10 * N)
    with rf.Simulation(rf.Configuration(params(N, NoQI, velocity_mode=reuse, gmres_tol=1e-9), pos, ori)) as s:
        s.assemble_system()
        A, b = s.matrix(), s.rhs()
        s.solve_system()
        s.update_velocities()
        x, (V, W) = s.coeffs(), s.velocities()
    p = rfo.make_params(M, N=N, NoQI=NoQI, eps=1e-2)
    A_o, b_o = rfo.assemble_system(p, pos, ori)
    A_p, _ = rfo.assemble_system(p, pos * (1 + 2.0 ** -52), ori)
    tol = max(1e-9, 3 * np.abs(A_p - A_o).max() / np.abs(A_o).max())
    assert np.all(np.abs(A - A_o) <= 2.0 ** -23 * np.abs(A_o) + tol * np.abs(A_o).max())
    assert np.abs(b - b_o).max() <= tol * np.abs(b_o).max()
    V_o, W_o = rfo.velocities(p, pos, ori, x)
    scale = max(np.abs(V_o).max(), np.abs(W_o).max())
    assert np.abs(V - V_o).max() <= 1e-6 * scale
    assert np.abs(W - W_o).max() <= 1e-6 * scale


def test_without_the_block_buffer():
    """Too little device memory for the blocks: they go straight into A, the same bits."""
    M = 700
    pos, ori = suspension(M, 7)
    out = []
    for full in (False, True):
        with rf.Simulation(rf.Configuration(params(5, 8, velocity_mode=1), pos, ori)) as s:
            torch.cuda.empty_cache()
            free = torch.cuda.mem_get_info()[0]
            # 700 x 699 blocks of 1280 bytes are 597 MiB
            hold = torch.empty(free - (300 << 20), dtype=torch.uint8, device="cuda") if full else None
            s.assemble_system()
            out.append((s.matrix_rows(0, 300), s.rhs()))
            del hold
            torch.cuda.empty_cache()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
