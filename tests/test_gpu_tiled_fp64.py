"""GPU: the FP64 panel and trailing-update kernels of the tiled fronts against
a dense solve of the exported gain matrix.

`big_front_flops` is set so low that fronts of every size are tiled: one
column to several panels, last panels narrower than a tile, fronts without
rows below their pivots (roots), and chunks and update tiles with remainders.
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


@pytest.mark.parametrize("n_bus, flops", [(8, 1), (14, 1), (33, 1), (118, 1), (301, 1), (301, 2e3), (1201, 2e4)])
def test_tiled_fp64_fronts_solve_the_gain_system(n_bus, flops):
    g = SyntheticGrid(n_bus, int(round(1.4 * n_bus)), 0x7E00 + n_bus)
    e = Estimator()
    e.set_option("big_front_flops", flops)
    e.load_network(g)
    e.upload_model()
    assert e.schedule_info().panel_steps > 0
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
