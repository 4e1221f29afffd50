"""GPU: the FP64 front kernels against a dense product with the exported gain
matrix.

Tiled fronts: `big_front_flops` is set so low that fronts of every size are
tiled: one column to several panels, last panels narrower than a tile, fronts
without rows below their pivots (roots), and chunks and update tiles with
remainders.  Single-CTA fronts: `big_front_flops` so high that every front that
fits is one, `warp_fronts` off so that the narrowest are too, and
`flow_small_f` moves them between the 16- and the 32-column panels.
Tolerance: the backward error of an FP64 Cholesky solve, ||Gx - b|| <=
8 n eps ||G|| ||x|| (max norms; a few times the usual bound's n eps).
"""
import numpy as np
import pytest

from conftest import gpu_available
from grids import synthetic_state
from state_estimation_with_cuda_gb300 import Estimator
from state_estimation_with_cuda_gb300.workloads import SyntheticGrid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    if not gpu_available():
        pytest.fail("GPU tests need a CUDA device; the product has no CPU fallback")


def check_solve(n_bus, seed, **options):
    g = SyntheticGrid(n_bus, int(round(1.4 * n_bus)), seed)
    e = Estimator()
    for k, v in options.items():
        e.set_option(k, v)
    e.load_network(g)
    e.upload_model()
    info = e.schedule_info()
    e.evaluate_at(*synthetic_state(g))
    rows, cols, vals = e.gain()
    n = 2 * n_bus - 1
    G = np.zeros((n, n))
    G[rows, cols] = vals
    G[cols, rows] = vals
    rhs = np.random.default_rng(n_bus).standard_normal(n)
    x = e.factor_solve(rhs)
    e.close()
    assert np.abs(G @ x - rhs).max() <= 8 * n * np.finfo(float).eps * np.abs(G).sum(axis=1).max() * np.abs(x).max()
    return info


@pytest.mark.parametrize("n_bus, flops", [(8, 1), (14, 1), (33, 1), (118, 1), (301, 1), (301, 2e3), (1201, 2e4)])
def test_tiled_fp64_fronts_solve_the_gain_system(n_bus, flops):
    assert check_solve(n_bus, 0x7E00 + n_bus, big_front_flops=flops).panel_steps > 0


@pytest.mark.parametrize("flow_small_f", [8, 32, 64, 128])
@pytest.mark.parametrize("n_bus", [8, 33, 118, 301, 1201, 2500])
def test_single_cta_fp64_fronts_solve_the_gain_system(n_bus, flow_small_f):
    info = check_solve(n_bus, 0x7F00 + n_bus, big_front_flops=1e18, warp_fronts=0, flow_small_f=flow_small_f)
    assert info.n_warp == 0 and info.n_phase_a + info.n_phase_b > 0
