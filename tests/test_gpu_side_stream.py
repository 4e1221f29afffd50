"""GPU: a level's single-CTA fronts on the side stream beside its tiled ones.

The fronts of a level do not touch each other's memory, so a step gives the
same bits however they overlap: solves repeated, captured in a graph and
launched directly, alone and in a batch.  FP64 grids whose levels hold both
kinds (`big_front_flops` moves the line between them), and the mixed pipeline
on a grid with tiled fronts.
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


def states(g, graphs, repeats, mixed, flops):
    e = Estimator()
    e.set_config(use_cuda_graphs=graphs)
    e.set_option("use_double_precision", int(not mixed))
    e.set_option("big_front_flops", flops)
    e.load_network(g)
    e.upload_model()
    out = []
    for _ in range(repeats):
        e.solve_with(max_iterations=4, tolerance=1e-30, flat_start=True)
        out.append(np.concatenate(e.voltages()))
    e.close()
    return out


@pytest.mark.parametrize("n_bus, mixed, flops", [(1000, False, 1e3), (3000, False, 3e4), (12000, False, 1e5),
                                                 (30000, True, 1e5)])
def test_side_stream_gives_the_same_bits(n_bus, mixed, flops):
    g = SyntheticGrid(n_bus, int(round(1.4 * n_bus)), 0x8600 + n_bus)
    ref, *more = states(g, 1, 8, mixed, flops)
    assert np.isfinite(ref).all()
    assert all(np.array_equal(ref, x) for x in more + states(g, 0, 3, mixed, flops))
    b = BatchEstimator(mixed=mixed)
    b.set_option("big_front_flops", flops)
    ids = [b.add_grid(x) for x in (SyntheticGrid(400, 560, 0x8500), g, SyntheticGrid(900, 1260, 0x8501))]
    for loop in (1, 0):
        b.set_option("device_loop", loop)
        b.solve(flat_start=True, max_iterations=4, tolerance=1e-30)
        x = np.concatenate(b.state(ids[1]))
        assert np.abs(x - ref).max() <= 1e-12  # same operations; the objective's sums aside
    b.close()
