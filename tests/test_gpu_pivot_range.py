"""GPU: FP64 pivots outside the range in which the kernels seed a reciprocal (or
square root) in FP32, on all four front paths, against a dense product with the
exported gain matrix.

Grids with scaled sigmas and branch impedances: pivots of 2^-110 to 2^-93 (on
both sides of the lower line at 2^-100), of 2^106 to 2^121 (above the upper one),
and of 2^-1042 to 2^-1012, more than half of them below 2^-1024, whose reciprocal
is infinite.

Tolerance, with G, x and b brought back to ordinary size by the power of two: the
backward error of an FP64 Cholesky solve, 8 n eps ||G|| ||x|| (max norms), and
for subnormal numbers half of 2^-1074 per operation: fewer than 2 n of them on
each entry of a row of G (n entries) and of b, n^2 2^-1074 (||x|| + 1).
"""
import numpy as np
import pytest

from conftest import gpu_available
from grids import copy_grid, synthetic_state
from state_estimation_with_cuda_gb300 import Estimator
from state_estimation_with_cuda_gb300.workloads import SyntheticGrid

pytestmark = pytest.mark.gpu

PATHS = {"warp": dict(warp_fronts=1, big_front_flops=1e18), "phase A": dict(warp_fronts=0, big_front_flops=1e18),
         "phase B": dict(warp_fronts=0, big_front_flops=1e18, flow_small_f=8),
         "level": dict(warp_fronts=0, big_front_flops=1e18, dataflow=0), "tiled": dict(warp_fronts=0, big_front_flops=1)}


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    if not gpu_available():
        pytest.fail("GPU tests need a CUDA device; the product has no CPU fallback")


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("n_bus", [118, 301])
@pytest.mark.parametrize("sigma, impedance", [(60, 0), (514, 10), (None, -14)])
def test_pivots_outside_the_fp32_range(sigma, impedance, n_bus, path):
    g = copy_grid(SyntheticGrid(n_bus, int(round(1.4 * n_bus)), 0x9A00 + n_bus))
    k = sigma or 0
    g.m_sigma = np.full(g.n_meas, 1e-12) if sigma is None else g.m_sigma * 2.0 ** k
    g.br_r, g.br_x = g.br_r * 2.0 ** impedance, g.br_x * 2.0 ** impedance
    e = Estimator()
    for key, value in PATHS[path].items():
        e.set_option(key, value)
    e.load_network(g)
    e.upload_model()
    e.evaluate_at(*synthetic_state(g))
    rows, cols, vals = e.gain()
    n = 2 * n_bus - 1
    G = np.zeros((n, n))
    G[rows, cols] = np.ldexp(vals, 2 * k)
    G[cols, rows] = np.ldexp(vals, 2 * k)
    rhs = np.random.default_rng(n_bus).standard_normal(n)
    x = e.factor_solve(np.ldexp(rhs, -2 * k))
    e.close()
    size = np.abs(x).max()
    bound = 8 * n * np.finfo(float).eps * np.abs(G).sum(axis=1).max() * size
    assert np.abs(G @ x - rhs).max() <= bound + n * n * np.ldexp(1.0, 2 * k - 1074) * (size + 1)
