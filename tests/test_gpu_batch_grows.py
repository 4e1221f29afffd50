"""GPU: a model that grows after it was uploaded.

The device arrays are as long as at the upload.  Reading states and results in
between has to give the uploaded network's estimates and the added elements'
start values, and the re-upload has to take both as its hot start, whatever was
read before.  The added grid is much larger than the uploaded ones, the reads
come in all orders, and each result is that of a handle which had the grid from
the beginning (equal bits: a grid's result does not depend on the batch).
"""
import numpy as np
import pytest

from conftest import gpu_available
from state_estimation_with_cuda_gb300 import BatchEstimator, Estimator, api
from state_estimation_with_cuda_gb300.workloads import SyntheticGrid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    if not gpu_available():
        pytest.fail("GPU tests need a CUDA device; the product has no CPU fallback")


def batch(mixed, *grids):
    b = BatchEstimator(mixed=mixed)
    for g in grids:
        b.add_grid(g)
    return b


def states(b, order):
    return {i: np.concatenate(b.state(i)) for i in order}


def start_state(g):
    return np.concatenate([g.v_setpoint, np.zeros(g.n_bus)])


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("order", [(0, 1, 2), (2, 1, 0), (1, 0, 1, 2), (2,), ()])
def test_states_and_hot_start_when_a_grid_is_added_after_a_solve(order, mixed):
    small = [SyntheticGrid(n, int(round(1.4 * n)), 0x9500 + n) for n in (30, 71)]
    large = SyntheticGrid(20000, 28000, 0x9501)
    want, hot = [], []
    for g in small:
        a = batch(mixed, g)
        a.solve(flat_start=True)
        want.append(np.concatenate(a.state(0)))
        r = a.solve(flat_start=False)[0]
        hot.append((r.status, r.iterations, np.concatenate(a.state(0))))
        a.close()
    a = batch(mixed, large)
    want.append(start_state(large))
    r = a.solve(flat_start=False)[0]
    hot.append((r.status, r.iterations, np.concatenate(a.state(0))))
    a.close()

    b = batch(mixed, *small)
    b.solve(flat_start=True)
    assert b.add_grid(large) == 2
    for i, x in states(b, order).items():
        assert np.array_equal(x, want[i]), i
    res = b.solve(flat_start=False)
    for i in (1, 2, 0):
        assert (res[i].status, res[i].iterations) == hot[i][:2]
        assert np.array_equal(np.concatenate(b.state(i)), hot[i][2]), i
    b.close()


def test_results_of_one_grid_when_elements_are_added_after_a_solve():
    """The added bus (on a new branch, unmeasured) reads as its start state, the
    others as estimated; injections and flows are those of the uploaded
    network; the next solve takes the new model."""
    g = SyntheticGrid(300, 420, 0x9502)
    e = Estimator()
    e.load_network(g)
    rc, _ = e.solve_with(max_iterations=20, tolerance=1e-6, flat_start=True)
    assert rc == 0
    v, th = e.voltages()
    flows, r = e.branch_flows(), e.residuals()
    e.evaluate_at(v, th)  # the same state, not read back yet
    n_new = 2000
    for i in range(n_new):
        e.add_bus("new%d" % i, type=api.BUS_PQ, v_setpoint=1.01)
        e.add_branch("line%d" % i, "BUS3" if i == 0 else "new%d" % (i - 1), "new%d" % i, 0.01, 0.05)
        e.add_measurement("m%d" % i, api.MEAS_V_MAG, "new%d" % i, 0.004)
        e.add_measurement("p%d" % i, api.MEAS_P_FLOW, "line%d" % i, 0.008)
        e.add_measurement("q%d" % i, api.MEAS_Q_FLOW, "line%d" % i, 0.008)
    v2, th2 = e.voltages()
    assert np.array_equal(v2[:300], v) and np.array_equal(th2[:300], th)
    assert np.array_equal(v2[300:], np.full(n_new, 1.01)) and not th2[300:].any()
    for x, y in zip(e.branch_flows(), flows):
        assert np.array_equal(x[:420], y)
    r2 = e.residuals()
    assert np.array_equal(r2[:g.n_meas], r) and not r2[g.n_meas:].any()
    z = np.concatenate([g.z, np.tile([1.0, 0.0, 0.0], n_new)])
    e.update_telemetry(z)
    rc, res = e.solve_with(max_iterations=20, tolerance=1e-6, flat_start=False)
    assert rc == 0 and res.status == 0
    assert len(e.voltages()[0]) == 300 + n_new
    e.close()
