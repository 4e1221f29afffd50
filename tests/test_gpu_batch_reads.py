"""GPU: telemetry set and states read grid by grid around batch solves.

Setting a grid's telemetry waits only for a copy of its own that may still be
running, and from the second read on the batch's states are served from one
copy; both must give what a handle of one grid gives, whatever the order:
telemetry set twice before a solve, one grid read, all read, read again after
another solve, after a whole-vector update and after a re-upload.  Equal bits
(a grid's result does not depend on the batch).
"""
import numpy as np
import pytest

from conftest import gpu_available
from state_estimation_with_cuda_gb300 import BatchEstimator
from state_estimation_with_cuda_gb300.workloads import SyntheticGrid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    if not gpu_available():
        pytest.fail("GPU tests need a CUDA device; the product has no CPU fallback")


def alone(g, z):
    b = BatchEstimator(mixed=True)
    b.add_grid(g, z)
    b.solve(flat_start=True)
    x = np.concatenate(b.state(0))
    b.close()
    return x


def test_states_read_in_any_order_are_the_last_solves():
    grids = [SyntheticGrid(n, int(round(1.4 * n)), 0x9100 + n) for n in (30, 71, 150, 301)]
    z = [[g.z.copy(), g.renoise(1, 1.0).copy(), g.renoise(2, 1.0).copy()] for g in grids]
    want = [[alone(g, zz) for zz in zs] for g, zs in zip(grids, z)]
    b = BatchEstimator(mixed=True)
    for g, zs in zip(grids, z):
        b.add_grid(g, zs[0])
    b.upload_model()

    def check(order, u):
        for i in order:
            assert np.array_equal(np.concatenate(b.state(i)), want[i][u]), (i, u)

    b.solve(flat_start=True)
    check([2], 0)  # one grid alone
    for i, zs in enumerate(z):
        b.set_telemetry(i, zs[2])
        b.set_telemetry(i, zs[1])  # the second overwrites the first
    check([3, 0, 1, 2], 0)  # still the first solve's
    b.solve(flat_start=True)
    check([1, 1, 0, 2, 3], 1)
    b.update_telemetry(np.concatenate([zs[0] for zs in z]))
    b.set_telemetry(1, z[1][2])
    b.solve(flat_start=True)
    check([0, 2], 0)
    check([1], 2)
    b.upload_model()
    check([0, 2, 3], 0)
    b.close()
