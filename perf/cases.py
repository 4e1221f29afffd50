"""What this library's users have it do, as cases that can be timed and compared.

A case is one pass through the public Python mirror of the C interface: host
arrays in (telemetry snapshots, states, right-hand sides), host arrays out
(|V| and theta, residuals, flows), as a control-room program sees it.  The
handle with its uploaded model is what such a program keeps; the telemetry of a
snapshot is not on the device before the pass.

  estimate  one grid: the snapshot's first estimate from a flat start, then
            `scans` tracking scans (1 % of the rows re-measured) hot-started
            from the previous estimate.  `report` reads every result back.
  breaker   one grid: a switch opens, the grid is estimated, the switch closes,
            the grid is estimated again.
  evaluate  the measurement layer: h(x), the Jacobian and the gradient at a state.
  linear    the linear layer: factorise G = H'WH and solve for a right-hand side.
  batch     many independent grids of 30 to 5000 buses in one call.
  served    a resident fleet: every grid submits a snapshot, all are awaited,
            twice.

Grids come from the repository's seeded generator with its default mix (|V| at
30 % of the buses, P+Q injection at 60 %, both-end P+Q flows on 70 % of the
branches, 1.4 branches per bus).  A case's size fixes its networks, as a
program's are fixed; the seed makes the telemetry, states and right-hand sides.
Precision: the plain FP64 pipeline ("fp64")
or the mixed one (FP32 factor, FP64 residual and state).
"""
import functools
import math

import numpy as np
import torch

from state_estimation_with_cuda_gb300 import BatchEstimator, Estimator, Server, SyntheticGrid
from state_estimation_with_cuda_gb300.workloads import fleet_sizes, grid_seed

MAX_ITERATIONS = 20
TOLERANCE = 1e-6
# The served fleet stops tighter: a grid hot-starts from whatever its last
# estimate was, so its answers repeat only as far as they are converged.
SERVED_TOLERANCE = 1e-9
SERVED_ITERATIONS = 40


def listed():
    return [
        # a feeder or a teaching network: latency of one call, everything read back
        dict(name="grid14_report_fp64", op="estimate", n=14, mixed=False, robust=False, scans=0, report=True),
        # a switching operation in a small transmission area
        dict(name="grid301_breaker_mixed", op="breaker", n=301, mixed=True),
        # Huber weights against 2 % gross errors, results reported
        dict(name="grid2003_robust_fp64", op="estimate", n=2003, mixed=False, robust=True, scans=0, report=True),
        # the tracking loop of a control area: first estimate, then four scans
        dict(name="grid10k_track_mixed", op="estimate", n=10000, mixed=True, robust=False, scans=4, report=False),
        # the drop-in precision on the same area
        dict(name="grid10k_flat_fp64", op="estimate", n=10000, mixed=False, robust=False, scans=0, report=False),
        # a national grid in the drop-in precision
        dict(name="grid60k_flat_fp64", op="estimate", n=60013, mixed=False, robust=False, scans=0, report=False),
        # the largest model the configuration allows for
        dict(name="grid200k_flat_mixed", op="estimate", n=200000, mixed=True, robust=False, scans=0, report=False),
        # measurement layer alone
        dict(name="evaluate_20k", op="evaluate", n=20011),
        # linear layer alone
        dict(name="linear_30k", op="linear", n=30011),
        # the batched workload (512 grids of 30 to 5000 buses)
        dict(name="batch512_mixed", op="batch", count=512, mixed=True),
        # a smaller batch in the drop-in precision
        dict(name="batch64_fp64", op="batch", count=64, mixed=False),
        # the served workload's size distribution, up to 20,000 buses
        dict(name="served40_mixed", op="served", count=40, hi=20000, mixed=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["estimate", "estimate", "estimate", "breaker", "evaluate", "linear", "batch", "served"])
    mixed = rng.random() < 0.5
    if op == "estimate":
        robust = not mixed and rng.random() < 0.3
        scans = 0 if robust else rng.choice([0, 0, 1, 3])
        hi = 5000 if robust else 40000 if scans else 160000 if mixed else 60000
        return dict(op=op, n=_log_int(rng, 14, hi), mixed=mixed, robust=robust, scans=scans, report=rng.random() < 0.3)
    if op == "breaker":
        return dict(op=op, n=_log_int(rng, 120, 30000), mixed=mixed)
    if op == "evaluate":
        return dict(op=op, n=_log_int(rng, 100, 100000))
    if op == "linear":
        return dict(op=op, n=_log_int(rng, 100, 60000))
    if op == "batch":
        return dict(op=op, count=_log_int(rng, 4, 400 if mixed else 128), mixed=mixed)
    return dict(op=op, count=rng.randint(8, 48), hi=_log_int(rng, 1000, 20000), mixed=mixed)


# --------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=600)
def _grid(n, gross=0.0, i=0):
    return SyntheticGrid(n, int(round(1.4 * n)), grid_seed(0x9E00 + n, i + 1), gross=gross)


def _telemetry(g, seed, scans=0):
    """A snapshot with fresh noise on every row (gross errors stay where they
    are), then `scans` more, each re-measuring 1 % of the rows of the one before."""
    gross = g.gross != 0
    err = np.where(gross, _gross_errors(g), 0.0)
    base = 1000 * (int(seed) % 2000000) + 1
    z = [g.renoise(base, 1.0).copy()]
    for u in range(scans):
        z.append(g.renoise(base + 1 + u, 0.01).copy())
    return [np.where(gross, g.h_true + err, x) for x in z]


def _gross_errors(g):
    if not hasattr(g, "gross_error"):
        g.gross_error = g.z - g.h_true
    return g.gross_error


def _state(g, seed):
    """A state near the operating point, as in the middle of a Gauss-Newton run."""
    r = np.random.default_rng(seed)
    v = g.v_true + 0.01 * r.standard_normal(g.n_bus)
    th = g.theta_true + 0.02 * r.standard_normal(g.n_bus)
    th[g.slack] = 0.0
    return v, th


def _handle(g, mixed):
    e = Estimator()
    if mixed:
        e.set_option("use_double_precision", 0)
    e.load_network(g)
    return e


def _batch_sizes(case):
    """Log-uniform over [30, 5000], as the batched workload's."""
    u = (np.arange(case["count"]) + 0.5) / case["count"]
    return [int(round(30 * (5000 / 30) ** x)) for x in u]


def _fleet_sizes(case):
    """The served fleet's Zipf(1.2) sizes over [30, hi], the largest always among them."""
    return fleet_sizes(case["count"] - 1, hi=case["hi"]) + [case["hi"]]


def _grids(case):
    sizes = _batch_sizes(case) if case["op"] == "batch" else _fleet_sizes(case)
    return [_grid(n, 0.0, i) for i, n in enumerate(sizes)]


@functools.lru_cache(maxsize=64)
def _switch_branch(n):
    """A branch a dispatcher can open: no bridge, no flow meters on it, both
    ends with other branches, and the grid still has an estimate without it."""
    g = _grid(n)
    for d in range(64):
        k = int(g._lib.segen_pick_nonbridge(g._h, d))
        if k < 0:
            continue
        e = _handle(g, False)
        e.add_switch("SW", "BR%d" % k, closed=False)
        e.upload_model()
        rc, r = e.solve_with(max_iterations=MAX_ITERATIONS, tolerance=TOLERANCE, flat_start=True)
        e.close()
        if rc == 0:
            return k
    raise ValueError("no branch of this grid can be opened")


def prepare(case, seed):
    op = case["op"]
    st = dict(case)
    if op in ("estimate", "breaker", "evaluate", "linear"):
        g = _grid(case["n"], 0.02 if case.get("robust") else 0.0)
        z = _telemetry(g, seed, case.get("scans", 0))
        e = _handle(g, case.get("mixed", False))
        if op == "breaker":
            e.add_switch("SW", "BR%d" % _switch_branch(case["n"]), closed=True)
        e.upload_model()
        st["e"] = e
        if op in ("estimate", "breaker"):
            st["z"] = z
        elif op == "evaluate":
            e.update_telemetry(z[0])
            st["x"] = _state(g, seed)
        else:
            e.evaluate_at(*_state(g, seed))
            st["rhs"] = np.random.default_rng([int(seed), 3]).standard_normal(2 * g.n_bus - 1)
        return st
    grids = _grids(case)
    st["z"] = [_telemetry(g, seed, 1 if op == "served" else 0) for g in grids]
    if op == "batch":
        b = BatchEstimator(mixed=case["mixed"])
        for g in grids:
            b.add_grid(g)
        b.upload_model()
        st["b"] = b
    else:
        s = Server(mixed=case["mixed"], max_iterations=SERVED_ITERATIONS, tolerance=SERVED_TOLERANCE)
        for g in grids:
            s.add_grid(g)
        s.start()
        st.update(s=s, sizes=[g.n_bus for g in grids])
    return st


# --------------------------------------------------------------------------- one pass
def _estimate(st):
    e, out = st["e"], []
    for k, z in enumerate(st["z"]):
        e.update_telemetry(z)
        rc, r = e.solve_with(max_iterations=MAX_ITERATIONS, tolerance=TOLERANCE, flat_start=k == 0,
                             robust=st["robust"])
        v, th = e.voltages()
        out.append(dict(status=r.status, iterations=r.iterations, v=v, th=th))
    if st["report"]:
        p, q = e.injections()
        pf, qf, pt, qt = e.branch_flows()
        flagged = np.zeros(len(st["z"][0]), np.int32)
        flagged[e.bad_data()] = 1
        out[-1].update(residuals=e.residuals(), p=p, q=q, pf=pf, qf=qf, pt=pt, qt=qt, objective=e.objective(),
                       flagged=flagged)
    return out


def _breaker(st):
    e, out = st["e"], []
    for closed in (False, True):
        e.set_switch("SW", closed)
        e.apply_switch_changes()
        e.update_telemetry(st["z"][0])
        rc, r = e.solve_with(max_iterations=MAX_ITERATIONS, tolerance=TOLERANCE, flat_start=True)
        v, th = e.voltages()
        out.append(dict(status=r.status, iterations=r.iterations, v=v, th=th))
    return out


def _batch(st):
    b = st["b"]
    for i, z in enumerate(st["z"]):
        b.set_telemetry(i, z[0])
    res = b.solve(flat_start=True, max_iterations=MAX_ITERATIONS, tolerance=TOLERANCE)
    vth = [b.state(i) for i in range(len(st["z"]))]
    return dict(status=np.array([r.status for r in res]), iterations=np.array([r.iterations for r in res]),
                v=np.concatenate([x[0] for x in vth]), th=np.concatenate([x[1] for x in vth]))


def _served(st):
    s, out = st["s"], []
    for u in (0, 1):
        bufs = [(np.empty(n), np.empty(n)) for n in st["sizes"]]
        tickets = [s.submit(i, z[u], out=bufs[i]) for i, z in enumerate(st["z"])]
        res = [s.wait(t) for t in tickets]
        out.append(dict(status=np.array([r.status for r in res]), v=np.concatenate([b[0] for b in bufs]),
                        th=np.concatenate([b[1] for b in bufs])))
    return out


def run(st):
    op = st["op"]
    if op == "estimate":
        return _estimate(st)
    if op == "breaker":
        return _breaker(st)
    if op == "evaluate":
        return st["e"].evaluate_at(*st["x"])
    if op == "linear":
        return st["e"].factor_solve(st["rhs"])
    if op == "batch":
        return _batch(st)
    return _served(st)


# --------------------------------------------------------------------------- work
# Per bus, from the generator's mix and the analysis of its grids: 5.46 rows,
# 25.2 Jacobian entries, 85 gain products, about 60 entries of L; one
# factorisation is about 1560 n (n / 2000)^0.45 operations.
ROWS, H_NNZ, PAIRS, L_NNZ = 5.46, 25.2, 85.0, 60.0
NETWORK_BYTES = 1.4 * (2 * 4 + 5 * 8 + 1) + ROWS * (3 * 4 + 8)  # branch and row data per bus
FLAT_STEPS, HOT_STEPS = 5, 4  # Gauss-Newton steps of a usual solve


def _factor_flops(n):
    return 1560.0 * n * (n / 2000.0) ** 0.45


def _step_flops(n):
    return n * (40.0 * H_NNZ + 2.0 * PAIRS + 4.0 * L_NNZ) + _factor_flops(n)


def work(case):
    op = case["op"]
    if op == "estimate":
        n, solves = case["n"], 1 + case["scans"]
        by = n * (NETWORK_BYTES + solves * (8 * ROWS + 16)) + (n * (8 * ROWS + 16 + 1.4 * 32) if case["report"] else 0)
        steps = MAX_ITERATIONS if case["robust"] else FLAT_STEPS + HOT_STEPS * case["scans"]
        return dict(bytes=by, flops=steps * _step_flops(n))
    if op == "breaker":
        n = case["n"]
        return dict(bytes=n * (NETWORK_BYTES + 8 * ROWS + 2 * 16), flops=2 * FLAT_STEPS * _step_flops(n))
    if op == "evaluate":
        n = case["n"]
        return dict(bytes=n * (NETWORK_BYTES + 16 + 8 * ROWS + (8 + 4) * H_NNZ + (8 + 4) * ROWS + 16),
                    flops=n * 40.0 * H_NNZ)
    if op == "linear":
        n = case["n"]
        return dict(bytes=n * ((8 + 4) * H_NNZ + 8 * ROWS + 4 * 8), flops=n * (2 * PAIRS + 4 * L_NNZ) + _factor_flops(n))
    sizes = _batch_sizes(case) if op == "batch" else _fleet_sizes(case)
    solves, steps = (1, FLAT_STEPS) if op == "batch" else (2, 2 * (HOT_STEPS + 2))
    return dict(bytes=sum(sizes) * (NETWORK_BYTES + solves * (8 * ROWS + 16)),
                flops=steps * sum(_step_flops(n) for n in sizes))


# --------------------------------------------------------------------------- the same in plain 64-bit arithmetic
class _Wls:
    """The weighted-least-squares estimate of one grid in numpy and torch: h(x)
    and its Jacobian row by row as sparse triples, the normal equations as a
    block-tridiagonal matrix over breadth-first levels of the grid, factorised
    block by block."""

    def __init__(self, g, status=None):
        self.g = g
        on = (np.asarray(g.br_status if status is None else status) != 0).astype(float)
        self.on = on
        d = np.maximum(g.br_r ** 2 + g.br_x ** 2, 1e-12)
        self.gs, self.bs = g.br_r / d, -g.br_x / d
        self.a = np.maximum(g.br_tap, 1e-12)
        self.bsf, self.bst = g.br_b / (2 * g.br_tap ** 2), g.br_b / 2
        n = g.n_bus
        f, t = g.br_from, g.br_to
        gs, bs, a, cs, sn = self.gs * on, self.bs * on, self.a, np.cos(g.br_shift), np.sin(g.br_shift)
        # off-diagonal Ybus entries, both directions, and the diagonal
        self.yi, self.yj = np.concatenate([f, t]), np.concatenate([t, f])
        self.yg = np.concatenate([-(gs * cs + bs * sn) / a, -(gs * cs - bs * sn) / a])
        self.yb = np.concatenate([-(-gs * sn + bs * cs) / a, -(gs * sn + bs * cs) / a])
        self.gd = np.bincount(f, gs / a ** 2, n) + np.bincount(t, gs, n)
        self.bd = np.bincount(f, bs / a ** 2 + self.bsf * on, n) + np.bincount(t, bs + self.bst * on, n)
        self.nth = n - 1
        bus = np.arange(n)
        self.cth = np.where(bus < g.slack, bus, bus - 1)
        self.cth[g.slack] = -1
        self.cv = self.nth + bus
        self.w = 1.0 / np.maximum(g.m_sigma, 1e-12) ** 2
        ty = g.m_type
        self.rows = {k: np.nonzero(np.isin(ty, v))[0] for k, v in
                     dict(v=(0,), p=(2, 7), q=(3, 8), pf=(4,), qf=(5,)).items()}
        if sum(len(r) for r in self.rows.values()) != g.n_meas:
            raise ValueError("a row type that the generator does not make")
        self._levels()

    def _levels(self):
        g, n = self.g, self.g.n_bus
        i, j = np.concatenate([g.br_from, g.br_to]), np.concatenate([g.br_to, g.br_from])
        o = np.argsort(i, kind="stable")
        ptr = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))])
        col = j[o]

        def bfs(root):
            lvl = np.full(n, -1)
            lvl[root] = 0
            front, d = np.array([root]), 0
            while len(front):
                cnt = ptr[front + 1] - ptr[front]
                at = np.repeat(ptr[front] - np.concatenate([[0], np.cumsum(cnt)[:-1]]), cnt) + np.arange(cnt.sum())
                front = np.unique(col[at])
                front = front[lvl[front] < 0]
                d += 1
                lvl[front] = d
            return lvl

        lvl = bfs(int(np.argmax(bfs(0))))
        if lvl.min() < 0:
            raise ValueError("grid in several islands")
        # a row couples buses up to two branches apart: blocks of two levels
        # couple with their neighbours only; thin ones are joined
        blk, size, of = np.bincount(lvl // 2), 0, []
        k = 0
        for s in blk:
            if size + s > 400 and size:
                k, size = k + 1, 0
            of.append(k)
            size += s
        b = np.array(of)[lvl // 2]
        order = np.argsort(b, kind="stable")
        states = np.concatenate([self.cth[order], self.cv[order]])
        sb = np.concatenate([b[order], b[order]])
        keep = states >= 0
        states, sb = states[keep], sb[keep]
        o2 = np.argsort(sb, kind="stable")
        self.states, sb = states[o2], sb[o2]
        self.pos = np.empty(len(self.states), np.int64)
        self.pos[self.states] = np.arange(len(self.states))
        self.bptr = np.concatenate([[0], np.cumsum(np.bincount(sb))])
        self.block_of = sb
        self.cost = float(np.sum(np.diff(self.bptr).astype(float) ** 3)) * 5

    def hx(self, v, th):
        """h(x) and the Jacobian as triples (row, state, value), sorted, repeated ones summed."""
        g = self.g
        n = g.n_bus
        th_ij = th[self.yi] - th[self.yj]
        c, s = np.cos(th_ij), np.sin(th_ij)
        vi, vj = v[self.yi], v[self.yj]
        gc, gq = self.yg * c + self.yb * s, self.yg * s - self.yb * c
        P = v * np.bincount(self.yi, vj * gc, n) + v ** 2 * self.gd
        Q = v * np.bincount(self.yi, vj * gq, n) - v ** 2 * self.bd
        h = np.zeros(g.n_meas)
        R, C, V = [], [], []

        def put(r, c_, x):
            k = c_ >= 0
            R.append(r[k]), C.append(c_[k]), V.append(np.broadcast_to(x, r.shape)[k])

        r = self.rows["v"]
        h[r] = v[g.m_loc[r]]
        put(r, self.cv[g.m_loc[r]], 1.0)
        o = np.argsort(self.yi, kind="stable")
        yptr = np.concatenate([[0], np.cumsum(np.bincount(self.yi, minlength=n))])
        for kind in ("p", "q"):
            r = self.rows[kind]
            b = g.m_loc[r]
            cnt = yptr[b + 1] - yptr[b]
            e = o[np.repeat(yptr[b] - np.concatenate([[0], np.cumsum(cnt)[:-1]]), cnt) + np.arange(cnt.sum())]
            rr, bb = np.repeat(r, cnt), np.repeat(b, cnt)
            if kind == "p":
                h[r] = P[b]
                dt, dv, own = vi * vj * gq, vi * gc, vj * gc
                diag_v, sign = 2 * v * self.gd, -1.0
            else:
                h[r] = Q[b]
                dt, dv, own = -vi * vj * gc, vi * gq, vj * gq
                diag_v, sign = -2 * v * self.bd, -1.0
            put(rr, self.cth[self.yj[e]], dt[e])
            put(rr, self.cv[self.yj[e]], dv[e])
            put(rr, self.cth[bb], sign * dt[e])
            put(rr, self.cv[bb], own[e])
            put(r, self.cv[b], diag_v[b])
            put(r, self.cth[b], 0.0)
        fl = self.flows(v, th, True)
        for kind, at in (("pf", 0), ("qf", 1)):
            for end in (0, 1):
                r = self.rows[kind]
                r = r[(g.m_end[r] != 0) == (end == 1)]
                k = g.m_loc[r]
                val, d = fl[2 * end + at]
                h[r] = val[k]
                i, j = g.br_from[k], g.br_to[k]
                put(r, self.cth[i], d[0][k]), put(r, self.cv[i], d[1][k])
                put(r, self.cth[j], -d[0][k]), put(r, self.cv[j], d[2][k])
        R, C, V = np.concatenate(R), np.concatenate(C), np.concatenate(V)
        key = R.astype(np.int64) * (2 * n) + C
        u, inv = np.unique(key, return_inverse=True)
        return h, u // (2 * n), u % (2 * n), np.bincount(inv.reshape(-1), V, len(u))

    def flows(self, v, th, derivatives=False):
        """P and Q at the from end, P and Q at the to end of every branch: values, with (d/dth_i, d/dV_i, d/dV_j) if wanted."""
        g = self.g
        i, j = g.br_from, g.br_to
        x = th[i] - th[j] - g.br_shift
        c, s, vi, vj, a, gs, bs, on = np.cos(x), np.sin(x), v[i], v[j], self.a, self.gs, self.bs, self.on
        fc, fs, tc, ts = gs * c + bs * s, gs * s - bs * c, gs * c - bs * s, gs * s + bs * c
        vals = [vi ** 2 / a ** 2 * gs - vi * vj / a * fc, -vi ** 2 / a ** 2 * (bs + self.bsf) - vi * vj / a * fs,
                vj ** 2 * gs - vi * vj / a * tc, -vj ** 2 * (bs + self.bst) + vi * vj / a * ts]
        if not derivatives:
            return [x * on for x in vals]
        ds = [(vi * vj / a * fs, 2 * vi / a ** 2 * gs - vj / a * fc, -vi / a * fc),
              (-vi * vj / a * fc, -2 * vi / a ** 2 * (bs + self.bsf) - vj / a * fs, -vi / a * fs),
              (vi * vj / a * ts, -vj / a * tc, 2 * vj * gs - vi / a * tc),
              (vi * vj / a * tc, vj / a * ts, -2 * vj * (bs + self.bst) + vi / a * ts)]
        return [(x * on, tuple(y * on for y in d)) for x, d in zip(vals, ds)]

    def injections(self, v, th):
        n = self.g.n_bus
        x = th[self.yi] - th[self.yj]
        c, s = np.cos(x), np.sin(x)
        return (v * np.bincount(self.yi, v[self.yj] * (self.yg * c + self.yb * s), n) + v ** 2 * self.gd,
                v * np.bincount(self.yi, v[self.yj] * (self.yg * s - self.yb * c), n) - v ** 2 * self.bd)

    def solve(self, R, C, V, w, b):
        """x with (H'WH) x = b."""
        p = self.pos[C]
        cnt = np.bincount(R, minlength=self.g.n_meas)
        start = np.concatenate([[0], np.cumsum(cnt)[:-1]])
        k = cnt[R]
        left = np.repeat(np.arange(len(R)), k)
        right = np.repeat(start[R] - np.concatenate([[0], np.cumsum(k)[:-1]]), k) + np.arange(k.sum())
        i, j, x = p[left], p[right], w[R[left]] * V[left] * V[right]
        low = self.block_of[i] >= self.block_of[j]
        i, j, x = i[low], j[low], x[low]
        bi, bj = self.block_of[i], self.block_of[j]
        nb = len(self.bptr) - 1
        o = np.argsort(2 * bi + (bi == bj), kind="stable")
        i, j, x, at = i[o], j[o], x[o], (2 * bi + (bi == bj))[o]
        cut = np.searchsorted(at, np.arange(2 * nb + 1))
        rhs = torch.from_numpy(b[self.states])
        L, M, y, keep = None, None, [], []
        for q in range(nb):
            r0, m = self.bptr[q], self.bptr[q + 1] - self.bptr[q]

            def block(t, c0, width):
                z = slice(cut[t], cut[t + 1])
                return torch.from_numpy(np.bincount((i[z] - r0) * width + (j[z] - c0), x[z], m * width).reshape(m, width))

            D, v = block(2 * q + 1, r0, m), rhs[r0:r0 + m].clone()
            if q:
                c0 = self.bptr[q - 1]
                M = torch.linalg.solve_triangular(L, block(2 * q, c0, r0 - c0).T, upper=False).T
                D, v = D - M @ M.T, v - M @ y[-1]
            L = torch.linalg.cholesky(D)
            y.append(torch.linalg.solve_triangular(L, v[:, None], upper=False)[:, 0])
            keep.append((L, M))
        out = [None] * nb
        for q in range(nb - 1, -1, -1):
            v = y[q]
            if q + 1 < nb:
                v = v - keep[q + 1][1].T @ out[q + 1]
            out[q] = torch.linalg.solve_triangular(keep[q][0].T, v[:, None], upper=True)[:, 0]
        res = np.empty(len(self.states))
        res[self.states] = torch.cat(out).numpy()
        return res

    def gradient(self, R, C, V, wr):
        return np.bincount(C, V * wr[R], 2 * self.g.n_bus - 1)

    def estimate(self, z, v, th, tolerance, limit, robust=False, gamma=1.5):
        for _ in range(limit):
            h, R, C, V = self.hx(v, th)
            r = z - h
            w = self.w
            if robust:
                sg = self.g.m_sigma
                w = np.where(np.abs(r / sg) <= gamma, w, gamma / (sg * np.abs(r) + 1e-12))
            dx = self.solve(R, C, V, w, self.gradient(R, C, V, w * r))
            k = self.cth >= 0
            th, v = th.copy(), np.clip(v + dx[self.cv], 0.5, 1.5)
            th[k] += dx[self.cth[k]]
            if np.abs(dx).max() < tolerance:
                break
        return v, th

    def flat(self):
        g = self.g
        return np.where(np.isin(g.bus_type, (1, 2)), g.v_setpoint, 1.0), np.zeros(g.n_bus)


MOST_COST = 2e12  # multiply-adds of the block factorisations of one exact()


def exact(case, seed):
    op = case["op"]
    if op in ("batch", "served"):
        if case["count"] > 64:
            return None
        grids = _grids(case)
        models = [_Wls(g) for g in grids]
        if sum(m.cost for m in models) * (24 if op == "served" else 5) > MOST_COST:
            return None
        zs = [_telemetry(g, seed, 1 if op == "served" else 0) for g in grids]
        out, x = [], [m.flat() for m in models]
        for u in range(len(zs[0])):
            tol, limit = (TOLERANCE, MAX_ITERATIONS) if op == "batch" else (SERVED_TOLERANCE / 100, SERVED_ITERATIONS)
            x = [m.estimate(z[u], *s, tol, limit) for m, z, s in zip(models, zs, x)]
            out.append(dict(status=None, v=np.concatenate([a for a, _ in x]), th=np.concatenate([t for _, t in x])))
        return dict(out[0], iterations=None) if op == "batch" else out
    robust = bool(case.get("robust"))
    g = _grid(case["n"], 0.02 if robust else 0.0)
    zs = _telemetry(g, seed, case.get("scans", 0))
    m = _Wls(g)
    if op == "evaluate":
        h, R, C, V = m.hx(*_state(g, seed))
        return dict(h_ptr=None, h_col=None, h_val=V, hx=h, rhs=m.gradient(R, C, V, m.w * (zs[0] - h)))
    if op == "linear":
        if m.cost > MOST_COST:
            return None
        _, R, C, V = m.hx(*_state(g, seed))
        return m.solve(R, C, V, m.w, np.random.default_rng([int(seed), 3]).standard_normal(2 * g.n_bus - 1))
    solves = 2 if op == "breaker" else 1 + case["scans"]
    if m.cost * (MAX_ITERATIONS if robust else 5 * solves) > MOST_COST:
        return None
    out = []
    if op == "breaker":
        for closed in (0, 1):
            status = g.br_status.copy()
            status[_switch_branch(case["n"])] = closed
            m = _Wls(g, status)
            v, th = m.estimate(zs[0], *m.flat(), TOLERANCE, MAX_ITERATIONS)
            out.append(dict(status=None, iterations=None, v=v, th=th))
        return out
    x = m.flat()
    for z in zs:
        x = m.estimate(z, *x, TOLERANCE, MAX_ITERATIONS, robust)
        out.append(dict(status=None, iterations=None, v=x[0], th=x[1]))
    if case["report"]:
        r = zs[-1] - m.hx(*x)[0]
        p, q = m.injections(*x)
        pf, qf, pt, qt = m.flows(*x)
        out[-1].update(residuals=r, p=p, q=q, pf=pf, qf=qf, pt=pt, qt=qt, objective=float(np.sum(m.w * r * r)),
                       flagged=None)
    return out
