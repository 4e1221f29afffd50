"""GPU: rows of the evaluation that ordinary grids do not have, in both
evaluation kernels (a thread per row; P rows with their Q twins), against the
oracle: branches that end where they start (their derivatives meet in one H
entry, their Ybus entries in the diagonal), and open branches with states so
large, infinite or NaN that the flow is not finite (0 x infinity is NaN, as in
the formulas).  Tolerances as for every row: 1e-12 of the value or the largest
derivative, 1e-10 for the gradient.
"""
import numpy as np
import pytest

from conftest import gpu_available
from grids import copy_grid, synthetic_state
from oracle.binding import Oracle
from state_estimation_with_cuda_gb300 import Estimator
from state_estimation_with_cuda_gb300.workloads import SyntheticGrid

pytestmark = pytest.mark.gpu

PAIR_ROWS = [0, 1 << 18]  # eval_pair_rows: pairs from the first row on, rows


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    if not gpu_available():
        pytest.fail("GPU tests need a CUDA device; the product has no CPU fallback")


def with_flow_rows(g, branches):
    """P, Q and |I| rows at both ends of the branches, appended."""
    n = len(branches)
    g.m_type = np.concatenate([g.m_type, np.tile(np.array([4, 5, 4, 5, 6, 6], np.int32), n)])
    g.m_loc = np.concatenate([g.m_loc, np.repeat(np.asarray(branches, np.int32), 6)])
    g.m_end = np.concatenate([g.m_end, np.tile(np.array([0, 0, 1, 1, 0, 1], np.int32), n)])
    g.m_sigma = np.concatenate([g.m_sigma, np.full(6 * n, 0.008)])
    g.z = np.concatenate([g.z, np.full(6 * n, 0.1)])
    g.n_meas = len(g.m_type)
    return g


def evaluate(g, v, th, exact, pair_rows):
    e = Estimator()
    e.set_option("eval_pair_rows", pair_rows)
    e.load_network(g)
    e.upload_model()
    got = e.evaluate_at(v, th, exact=exact)
    flows = e.branch_flows()
    e.close()
    o = Oracle(g)
    ref = o.evaluate(v, th, g.z, exact=exact)
    res = o.results(v, th)
    o.close()
    assert np.array_equal(got["h_ptr"], ref["h_ptr"]) and np.array_equal(got["h_col"], ref["h_col"])
    return got, ref, flows, res


@pytest.mark.parametrize("pair_rows", PAIR_ROWS)
@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("n_bus", [14, 301])
def test_branches_that_end_where_they_start(n_bus, exact, pair_rows):
    g = copy_grid(SyntheticGrid(n_bus, int(round(1.4 * n_bus)), 0x9B00 + n_bus))
    inj = g.m_loc[np.isin(g.m_type, (2, 3))]
    buses = [g.slack, int(inj[0]), int(inj[-1]), int(inj[-1])]  # two at one bus
    k = np.arange(g.n_branch, g.n_branch + len(buses))
    for name, values in dict(br_from=buses, br_to=buses, br_r=[0.01, 0.02, 0.03, 0.02], br_x=[0.05, 0.1, 0.1, 0.2],
                             br_b=[0.02, 0.0, 0.03, 0.01], br_tap=[1.0, 0.96, 1.04, 1.0], br_shift=[0.0, 0.1, -0.2, 0.0],
                             br_status=[1, 1, 1, 1]).items():
        a = getattr(g, name)
        setattr(g, name, np.concatenate([a, np.asarray(values, a.dtype)]))
    g.n_branch += len(buses)
    with_flow_rows(g, k)
    got, ref, flows, res = evaluate(g, *synthetic_state(g), exact, pair_rows)
    assert np.allclose(got["hx"], ref["hx"], rtol=1e-12, atol=1e-12)
    assert np.allclose(got["h_val"], ref["h_val"], rtol=1e-12, atol=1e-12 * np.abs(ref["h_val"]).max())
    assert np.allclose(got["rhs"], ref["rhs"], rtol=1e-10, atol=1e-10 * np.abs(ref["rhs"]).max())
    for f, want in zip(flows, res[2:]):
        assert np.allclose(f, want, rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("pair_rows", PAIR_ROWS)
@pytest.mark.parametrize("bad", [None, 1e200, np.inf, np.nan])
def test_open_branches(bad, pair_rows):
    g = copy_grid(SyntheticGrid(301, 421, 0x9C01))
    k = np.arange(3, g.n_branch, 7)
    g.br_status[k] = 0
    rows = np.arange(g.n_meas, g.n_meas + 6 * len(k))
    with_flow_rows(g, k)
    v, th = synthetic_state(g)
    if bad is not None:
        v[g.br_from[k[::3]]] = bad
        v[g.br_to[k[1::3]]] = bad
    got, ref, _, _ = evaluate(g, v, th, True, pair_rows)
    if bad is None:  # every row; else the open branches' (others' infinities meet in an order of their own)
        rows = np.arange(g.n_meas)
        assert np.allclose(got["rhs"], ref["rhs"], rtol=1e-10, atol=1e-10 * np.abs(ref["rhs"]).max())
    h = np.concatenate([np.arange(ref["h_ptr"][q], ref["h_ptr"][q + 1]) for q in rows])
    scale = np.abs(ref["h_val"][h][np.isfinite(ref["h_val"][h])]).max()
    assert np.allclose(got["hx"][rows], ref["hx"][rows], rtol=1e-12, atol=1e-12, equal_nan=True)
    assert np.allclose(got["h_val"][h], ref["h_val"][h], rtol=1e-12, atol=1e-12 * scale, equal_nan=True)
    if bad is not None:
        assert np.isnan(ref["hx"][rows]).any() and not np.isnan(ref["hx"][rows]).all()
