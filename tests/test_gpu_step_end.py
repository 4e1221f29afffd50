"""GPU: the end of a Gauss-Newton step, where the update's last CTA takes the
maximum over all CTAs and decides.

max |dx| of the one step from a flat start against the difference of the
states (FP64 and mixed): equal up to the rounding of x + dx, half an ulp of
the largest state and of the difference.  Sizes: one CTA of 256 buses, its
edges, and more CTAs (70,000 buses: 274) than the last one has threads.  In a
batch: more grids than a CTA has threads, grids of one, two and three items
of 2,048 buses; results against each grid alone (same operations).
"""
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


def one(g, mixed, max_iterations=20):
    e = Estimator()
    e.set_option("use_double_precision", int(not mixed))
    e.set_config(voltage_min_pu=-1e3, voltage_max_pu=1e3)  # no clamp
    e.load_network(g)
    e.upload_model()
    _, r = e.solve_with(max_iterations=max_iterations, tolerance=1e-6, flat_start=True)
    out = r.iterations, r.max_mismatch, *e.voltages()
    e.close()
    return out


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("n_bus", [14, 255, 256, 257, 70000])
def test_largest_step_entry(n_bus, mixed):
    g = SyntheticGrid(n_bus, int(round(1.4 * n_bus)), 0x8300 + n_bus)
    _, mm, v, th = one(g, mixed, max_iterations=1)
    v0 = np.where(np.asarray(g.bus_type) == 0, 1.0, g.v_setpoint)
    step = max(np.abs(v - v0).max(), np.abs(th).max())
    assert abs(mm - step) <= 2.0 ** -52 * max(np.abs(v).max(), np.abs(th).max(), 1.0)


@pytest.mark.parametrize("mixed", [True, False])
def test_batch_of_more_grids_than_a_block_has_threads(mixed):
    sizes = [30 + i % 7 for i in range(300)] + [2048, 2049, 4097]
    grids = [SyntheticGrid(n, int(round(1.4 * n)), 0x8400 + i) for i, n in enumerate(sizes)]
    out = []
    for loop in (1, 0):
        b = BatchEstimator(mixed=mixed)
        b.set_option("device_loop", loop)
        b.set_config(voltage_min_pu=-1e3, voltage_max_pu=1e3)
        for g in grids:
            b.add_grid(g)
        res = b.solve(flat_start=True, max_iterations=20, tolerance=1e-6)
        out.append([(r.status, r.iterations, r.max_mismatch) for r in res])
        b.close()
    assert out[0] == out[1]
    for i in (0, 255, 256, 299, 300, 301, 302):
        its, mm, _, _ = one(grids[i], mixed)
        assert out[0][i][:2] == (0, its)
        assert abs(out[0][i][2] - mm) <= 1e-12
