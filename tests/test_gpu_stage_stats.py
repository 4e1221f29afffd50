"""GPU: the stage statistics with profiling on.  Every stage of a step is timed,
the right-hand side too, and the estimates are those without profiling (equal
bits: the same operations, b in a launch of its own)."""
import numpy as np
import pytest

from conftest import gpu_available
from state_estimation_with_cuda_gb300 import BatchEstimator, Estimator
from state_estimation_with_cuda_gb300.workloads import SyntheticGrid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    if not gpu_available():
        pytest.fail("GPU tests need a CUDA device; the product has no CPU fallback")


def check(st, steps):
    for stage in range(5):  # 0 evaluate, 1 factorisation, 2 right-hand side, 3 solves, 4 update
        assert st.calls[stage] == steps and st.launches[stage] >= steps and st.ms[stage] > 0.0, stage


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("robust", [False, True])
@pytest.mark.parametrize("n_bus", [14, 2500])
def test_every_stage_of_a_grids_steps_is_timed(n_bus, robust, mixed):
    g = SyntheticGrid(n_bus, int(round(1.4 * n_bus)), 0x9800 + n_bus)
    out = []
    for profiling in (0, 1):
        e = Estimator()
        e.set_option("use_double_precision", int(not mixed))
        e.set_config(enable_profiling=profiling)
        e.load_network(g)
        _, r = e.solve_with(max_iterations=8, tolerance=1e-6, flat_start=True, robust=robust)
        if profiling:
            check(e.stats(), r.iterations)
        out.append((r.status, r.iterations, r.max_mismatch, *np.concatenate(e.voltages())))
        e.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("mixed", [True, False])
def test_every_stage_of_a_batchs_steps_is_timed(mixed):
    grids = [SyntheticGrid(n, int(round(1.4 * n)), 0x9900 + n) for n in (30, 301, 1201)]
    out = []
    for profiling in (0, 1):
        b = BatchEstimator(mixed=mixed)
        b.set_config(enable_profiling=profiling)
        for g in grids:
            b.add_grid(g)
        res = b.solve(flat_start=True)
        if profiling:
            check(b.stats(), max(r.iterations for r in res))
        out.append([(r.status, r.iterations, r.max_mismatch, *np.concatenate(b.state(i))) for i, r in enumerate(res)])
        b.close()
    assert out[0] == out[1]
