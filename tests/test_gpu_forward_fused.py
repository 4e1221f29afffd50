"""GPU: the forward substitution that the factorisation carries along against
the forward sweep.

With `gain_policy` 1 the first step of a solve factorises (and carries the
right-hand side along); a second solve from the same flat start reuses that
factor, so its first step runs the forward sweep on the same right-hand side.
FP32 does the same operations in the same order both ways: equal bits.  FP64
solves L y = b by rows in the factorisation and by columns in the sweep:
states within 1e-10 (the FP64 solve itself is good to about 1e-12 on these
grids).

Sizes: warp fronts alone, the two single-CTA phases, tiled fronts (mixed:
30,000 buses; FP64 from 2,500 on), with and without the warp phase.
"""
import numpy as np
import pytest

from conftest import gpu_available
from state_estimation_with_cuda_gb300 import Estimator
from state_estimation_with_cuda_gb300.workloads import SyntheticGrid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    if not gpu_available():
        pytest.fail("GPU tests need a CUDA device; the product has no CPU fallback")


SIZES = [(14, 1), (33, 0), (301, -1), (301, 0), (2500, -1), (10000, -1), (30000, -1)]


@pytest.mark.parametrize("n_bus, warp, mixed, tile_flow",
                         [(n, w, m, 0) for n, w in SIZES for m in (True, False)] + [(30000, -1, True, 1)])
def test_carried_forward_substitution_equals_the_sweep(n_bus, warp, mixed, tile_flow):
    g = SyntheticGrid(n_bus, int(round(1.4 * n_bus)), 0x8100 + n_bus)
    e = Estimator()
    for k, v in dict(use_double_precision=int(not mixed), gain_policy=1, warp_fronts=warp, tile_flow=tile_flow).items():
        e.set_option(k, v)
    e.load_network(g)
    e.upload_model()
    states = []
    for _ in range(2):
        e.solve_with(max_iterations=1, tolerance=1e-12, flat_start=True)
        states.append(np.concatenate(e.voltages()))
    st = e.stats()
    e.close()
    assert st.calls[1] == 1 and st.iterations == 2  # one factorisation, two steps
    if mixed:
        assert np.array_equal(states[0], states[1])
    else:
        assert np.abs(states[0] - states[1]).max() <= 1e-10
