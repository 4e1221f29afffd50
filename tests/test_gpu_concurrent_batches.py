"""GPU: FP64 batches solved side by side, over and over.

The panels of the FP64 fronts are handed from warp to warp in shared memory; with
other batches' CTAs on the same SMs the warps of a CTA are delayed in ways that
one batch alone does not show.  Every solve must end without a timed-out wait and
with the bits of the first.
"""
import threading

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


@pytest.mark.parametrize("dataflow", [1, 0])
def test_fp64_batches_side_by_side(dataflow):
    batches, first, errors = [], [], []
    for t, sizes in enumerate(([30, 71, 118, 301, 368] * 20, [500, 1201, 2500] * 6, [4000, 5000])):
        b = BatchEstimator(mixed=False)
        b.set_option("dataflow", dataflow)
        for i, n in enumerate(sizes):
            b.add_grid(SyntheticGrid(n, int(round(1.4 * n)), 0x9D00 + 1000 * t + i))
        b.solve(flat_start=True)
        first.append([np.concatenate(b.state(i)) for i in range(len(sizes))])
        batches.append(b)

    def run(k):
        try:
            for _ in range(60):
                res = batches[k].solve(flat_start=True)
                assert all(r.status == 0 for r in res)
            for i, x in enumerate(first[k]):
                assert np.array_equal(np.concatenate(batches[k].state(i)), x), (k, i)
        except Exception as e:  # reported by the test's thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(batches))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    [b.close() for b in batches]
    assert not errors, errors
