"""GPU: a batch engine's inner state, through tests/engine_probe.cpp."""
import ctypes
import os

import numpy as np
import pytest

from conftest import gpu_available
from state_estimation_with_cuda_gb300 import _build
from state_estimation_with_cuda_gb300.api import _grid_arrays
from state_estimation_with_cuda_gb300.workloads import SyntheticGrid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    if not gpu_available():
        pytest.fail("GPU tests need a CUDA device; the product has no CPU fallback")
    so = str(tmp_path_factory.mktemp("probe") / "engine_probe.so")
    objs = [os.path.join(_build.OBJ, rel.replace("/", "_") + ".o")
            for rel in _build.CORE_CU + _build.CORE_CPP if not rel.startswith(("api/", "serve/"))]
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "engine_probe.cpp")
    _build._run([_build.NVCC] + _build.ARCH + ["-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", so, src] + objs +
                ["-lcudart_static", "-ldl", "-lrt", "-lpthread"])
    lib = ctypes.CDLL(so)
    lib.probe_new.restype = ctypes.c_void_p
    return lib


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


class Batch:
    def __init__(self, lib, grids, mixed, dataflow):
        self.lib, self.grids = lib, grids
        self.e = ctypes.c_void_p(lib.probe_new(int(mixed), int(dataflow)))
        for i, g in enumerate(grids):
            a = _grid_arrays(g)
            assert lib.probe_add_grid(self.e, g.n_bus, ptr(a[0]), ptr(a[1]), g.n_branch, *map(ptr, a[2:10]), g.n_meas,
                                      *map(ptr, a[10:])) == i

    def solve(self, flat, tol=1e-6):
        steps = np.empty(len(self.grids), np.int32)
        assert self.lib.probe_solve(self.e, ptr(np.array(flat, np.uint8)), ctypes.c_double(tol), ptr(steps)) == 0
        return list(steps)

    def solution(self, i):
        x = np.empty(2 * self.grids[i].n_bus - 1)
        assert self.lib.probe_solution(self.e, i, ptr(x)) == 0
        return x

    def stream(self, i, tol=1e-6):
        assert self.lib.probe_stream(self.e, i, ctypes.c_double(tol)) == 0

    def state(self, i):
        v, th = np.empty(self.grids[i].n_bus), np.empty(self.grids[i].n_bus)
        assert self.lib.probe_state(self.e, i, ptr(v), ptr(th)) == 0
        return np.concatenate([v, th])

    def close(self):
        self.lib.probe_delete(self.e)


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("dataflow", [0, 1])
def test_solution_of_a_finished_grid_stays(probe, mixed, dataflow):
    """A grid that has converged takes no part in the batch's further steps: its
    solution vector stays that of its last step (as of the grid alone)."""
    grids = [SyntheticGrid(n, int(round(1.4 * n)), 0x9600 + n) for n in (71, 150, 301)]
    flat = [[1, 1, 1], [0, 1, 0]]
    b = Batch(probe, grids, mixed, dataflow)
    steps = [b.solve(f) for f in flat]
    assert steps[1][0] < steps[1][1]  # grid 0 stops first
    for i, g in enumerate(grids):
        a = Batch(probe, [g], mixed, dataflow)
        assert [a.solve([f[i]])[0] for f in flat] == [s[i] for s in steps]
        assert np.array_equal(b.solution(i), a.solution(0)), i
        a.close()
    b.close()


def test_states_come_in_one_copy_again_after_stream_mode(probe):
    """In stream mode each grid's state is read from the device, before and
    after it from one copy of the batch's states; the values are those of the
    grid alone each time."""
    grids = [SyntheticGrid(n, int(round(1.4 * n)), 0x9700 + n) for n in (30, 71, 150)]
    b = Batch(probe, grids, True, 1)
    alone = [Batch(probe, [g], True, 1) for g in grids]

    def check(shared):
        for i, a in enumerate(alone):
            assert np.array_equal(b.state(i), a.state(0)), i
        assert probe.probe_reads_shared(b.e) == shared

    b.solve([1, 1, 1])
    [a.solve([1]) for a in alone]
    check(1)
    for i in (1, 0, 1):
        b.stream(i, 1e-9)
        alone[i].stream(0, 1e-9)
        check(0)
    b.solve([0, 1, 0])
    [a.solve([f]) for a, f in zip(alone, (0, 1, 0))]
    check(1)
    b.stream(2, 1e-9)
    alone[2].stream(0, 1e-9)
    check(0)
    b.close()
    [a.close() for a in alone]
