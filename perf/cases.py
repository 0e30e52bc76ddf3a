"""The workloads this framework is timed on, each through its public entry points.

Four kinds of program use it:

* ``decompose``  the drop-in call: host columns in, ``prepare`` -> ``solve`` -> ``result`` -> ``release``
  out.  Nothing is kept between two passes; a pass pays for the whole path.
* ``shard``      a program that holds one prepared generation on the GPU and decomposes probe sets of
  its own seeds on it, as a rank of a probe-sharded run does: ``DeviceBackend.leverage`` (fit and
  leverage probes, accumulators in a CUDA tensor), ``target`` (adjustment and target probes) and
  ``finish``.  The library holds one generation at a time, so the passes of a case share it and
  differ by their probe seed.
* ``exact``      the exact-leverage estimator from host columns.
* ``train``      one forward and backward pass of the preconditioner's graph network.

Panels come from the repository's generator; the named sizes are the benchmark's own workloads (some
at a fraction of their workers), everything else is drawn.  The request keeps the library's default
tolerance, 1e-10.
"""

import numpy as np
import torch

from fevc_b200 import abi, learned, sharded
from fevc_b200.panel import generate_panel

BASE = dict(kind="decompose", workers=20_000, firms=1_000, periods=5, move_p=0.10, pareto=1.5, regions=1,
            cross_p=0.0, controls=False, deletion=1, probes=200, block=0, preconditioner=0, precision=0,
            numerical=False, columns=0)


def _case(name, **kw):
    return dict(BASE, name=name, **kw)


def listed():
    return [
        # a survey extract or a bootstrap replicate: launches and latencies are all there is
        _case("decompose_2k", workers=2_000, firms=150, move_p=0.20),
        # the 20,000-worker benchmark panel from host columns, the library's defaults
        _case("decompose_20k"),
        # leave-observation-out with year controls and the numerical covariance (mcse(all))
        _case("numerical_20k", controls=True, deletion=2, numerical=True),
        # exact leverages, the smaller-panel estimator
        _case("exact_4k", kind="exact", workers=4_000, firms=200, periods=6, move_p=0.08, pareto=1.3, probes=2),
        # a small panel decomposed again and again; an odd probe count leaves ragged last blocks
        _case("shard_20k_odd", kind="shard", probes=77),
        # 1M workers, year controls, 200 probes: the plain FP64 form
        _case("shard_1m_controls", kind="shard", workers=1_000_000, firms=50_000, controls=True),
        # one 100-probe set of the 3M-worker batched workload, FP64
        _case("shard_3m_sets", kind="shard", workers=3_000_000, firms=150_000, periods=6, move_p=0.08, pareto=1.3,
              probes=100),
        # the two-region workload at 0.2 of its workers, FP32 storage
        _case("shard_1m_regions", kind="shard", workers=1_000_000, firms=50_000, periods=6, regions=2, cross_p=0.001,
              probes=100, block=64, preconditioner=1, precision=1),
        # the 10M-worker workload at 0.2 of its workers: leave-observation-out, controls, the learned stage
        _case("shard_2m_learned", kind="shard", workers=2_000_000, firms=200_000, pareto=1.2, controls=True,
              deletion=2, probes=128, block=64, preconditioner=3, precision=1),
        # the same at 0.02 with a ragged probe count
        _case("shard_200k_learned", kind="shard", workers=200_000, firms=20_000, pareto=1.2, controls=True,
              deletion=2, probes=250, block=64, preconditioner=3, precision=1),
        # the aggregation-multigrid form a CMG request takes
        _case("shard_200k_cmg", kind="shard", workers=200_000, firms=10_000, probes=64, block=64, preconditioner=2),
        # one training pass on a panel of the default training size
        _case("train_20k", kind="train", firms=1_500, probes=2, columns=16),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["decompose", "decompose", "shard", "shard", "shard", "shard", "shard", "exact", "train"])
    top = {"decompose": 40_000, "shard": 1_000_000, "exact": 4_500, "train": 40_000}[kind]
    workers = log(1_500, top)
    c = dict(BASE, kind=kind, workers=workers, firms=2 * max(40, int(workers / rng.uniform(10, 25)) // 2),
             periods=rng.choice([4, 5, 5, 6]), move_p=round(rng.uniform(0.08, 0.2), 3),
             pareto=round(rng.uniform(1.2, 1.6), 2))
    if rng.random() < 0.15:
        c.update(regions=2, cross_p=0.01)
    if kind == "exact":
        return dict(c, probes=2)
    if kind == "train":
        return dict(c, probes=2, columns=rng.choice([8, 16, 32]))
    c.update(controls=rng.random() < 0.5, deletion=rng.choice([1, 2]), probes=log(100, 300))
    if kind == "decompose":
        return dict(c, numerical=rng.random() < 0.25)
    form = rng.choice(["default", "default", "mixed", "uniform", "learned", "learned", "narrow", "cmg"])
    if form == "mixed":
        c.update(block=64, preconditioner=1, precision=1)
    elif form == "uniform":
        c.update(block=rng.choice([32, 64]), preconditioner=4, precision=1)
    elif form == "learned":
        c.update(block=64, preconditioner=3, precision=rng.choice([0, 1]))
    elif form == "narrow":
        c.update(block=rng.choice([8, 16, 32]), preconditioner=1)
    elif form == "cmg":
        c.update(block=64, preconditioner=2, workers=min(workers, 200_000), probes=log(100, 128))
        c["firms"] = 2 * max(40, c["workers"] // 40)
    return c


# ---------------------------------------------------------------------------------------------------
# inputs and handles

_library = None
_held = {}  # the generation that the shard passes of one case share


def _lib():
    global _library
    if _library is None:
        _library = abi.load()
        learned.install(_library, learned.load_params())
    return _library


def _panel(case, seed):
    return generate_panel(case["workers"], case["firms"], case["periods"], move_p=case["move_p"],
                          pareto_shape=case["pareto"], year_controls=case["controls"], regions=case["regions"],
                          cross_p=case["cross_p"], deletion="observation" if case["deletion"] == 2 else "match",
                          seed=seed)


def _request(engine, case, seed):
    q = engine.default_request_v5(case["deletion"])
    v1 = q.v4.v3.v2.v1
    v1.seed, v1.probes, v1.maximum_iterations = seed, case["probes"], 20_000
    q.v4.v3.v2.algorithm = 2
    if case["deletion"] == 2 or case["controls"]:
        q.v4.v3.engine = 2
    return q


def _hold(case):
    """The prepared generation of this case, kept while its passes run."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _held.get("key") != key:
        _held.clear()
        panel = _panel(case, 20261203)
        e = abi.Engine(_lib())
        e.prepare(panel, deletion_mode=case["deletion"])
        e.device_options(case["block"], case["preconditioner"], case["precision"])
        _held.update(key=key, engine=e, controls=len(panel.controls))
    return _held["engine"], _held["controls"]


def prepare(case, seed):
    lib = _lib()
    if case["kind"] == "shard":
        engine, controls = _hold(case)
        q = _request(engine, case, 1 + seed)
        return {"case": case, "backend": sharded.DeviceBackend(engine, q, controls, torch.device("cuda"))}
    _held.clear()
    panel = _panel(case, seed)
    if case["kind"] == "train":
        t = learned.Trainer(lib, seed=1 + seed % 1000)
        t.add_panel(panel, columns=case["columns"], seed=seed)
        return {"case": case, "trainer": t}
    return {"case": case, "lib": lib, "panel": panel, "seed": 1 + seed}


def _components(res):
    return {k: np.array(v) for k, v in res.items()}


def run(state):
    case = state["case"]
    if case["kind"] == "shard":
        b = state["backend"]
        acc = b.leverage(0, case["probes"])
        draws = b.target(0, case["probes"], acc)
        return {"accumulators": acc, "draws": draws, **_components(b.finish(draws))}
    if case["kind"] == "train":
        loss, gradient = state["trainer"].gradient(0)
        return {"loss": np.float32(loss), "gradient": gradient}
    panel = state["panel"]
    e = abi.Engine(state["lib"])
    e.prepare(panel, deletion_mode=case["deletion"])
    out = {}
    if case["kind"] == "exact":
        e.exact_ceiling(1_000_000)
        e.solve_v5(e.exact_request_v5())
    else:
        q = _request(e, case, state["seed"])
        if case["numerical"]:
            e.solve_numerical(e.numerical_request(q, len(panel.controls)))
            num = e.numerical_result()
            out = {"status": int(num["status"]), "covariance": np.array(num["usable"]),
                   "mcse": np.array(num["mcse"])}
        else:
            e.solve_v5(q, len(panel.controls))
    out.update(_components(e.result()), retained=e.retained_mask(panel.rows))
    e.release()
    return out


def work(case):
    """Inputs read once and outputs written once; operations: one sparse product with every right-hand
    side (or one pass over the network's weights per vertex)."""
    rows = case["workers"] * case["periods"]
    if case["kind"] == "train":
        n = case["firms"]
        return {"bytes": 4.0 * n * (8 + 6 * case["columns"]) + 8.0 * 33_000, "flops": 6.0 * n * 26_000}
    columns = 6 + (case["periods"] - 1 if case["controls"] else 0)
    out = 0.0
    if case["kind"] == "shard":  # retained units or rows: movers, or all rows
        out = 64.0 * rows if case["deletion"] == 2 else 40.0 * rows * case["move_p"] * 1.5
    rhs = 2.0 * case["workers"] if case["kind"] == "exact" else 1.0 + 3.0 * case["probes"]
    return {"bytes": 8.0 * rows * columns + out, "flops": 4.0 * rows * rhs}


# ---------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain numpy and torch

def _low_points(n, eu, ev):
    """Articulation vertices and bridge edges of a simple graph (iterative depth-first search)."""
    order = np.argsort(np.concatenate([eu, ev]), kind="stable")
    ends = np.concatenate([ev, eu])[order].tolist()
    edge = (order % len(eu)).tolist()
    ptr = np.concatenate([[0], np.cumsum(np.bincount(np.concatenate([eu, ev]), minlength=n))]).tolist()
    seen, low, at = [0] * n, [0] * n, list(ptr[:n])
    via, cut, bridges, clock = [-1] * n, np.zeros(n, bool), [], 0
    for root in range(n):
        if seen[root] or ptr[root] == ptr[root + 1]:
            continue
        clock += 1
        seen[root] = low[root] = clock
        stack, children = [root], 0
        while stack:
            v = stack[-1]
            if at[v] < ptr[v + 1]:
                a = at[v]
                at[v] += 1
                u = ends[a]
                if edge[a] == via[v]:
                    continue
                if seen[u]:
                    low[v] = min(low[v], seen[u])
                else:
                    clock += 1
                    seen[u] = low[u] = clock
                    via[u] = edge[a]
                    children += v == root
                    stack.append(u)
            else:
                stack.pop()
                if stack:
                    p = stack[-1]
                    low[p] = min(low[p], low[v])
                    if low[v] > seen[p]:
                        bridges.append(via[v])
                    if p != root and low[v] >= seen[p]:
                        cut[p] = True
        cut[root] = children > 1
    return cut, np.array(bridges, dtype=np.int64)


def _largest(worker, firm, mass, on, workers, firms):
    """Of the edges `on`, those in the component with the most firms (then the most rows)."""
    label = np.arange(workers + firms)
    w, f = worker[on], workers + firm[on]
    while True:
        lo = np.minimum(label[w], label[f])
        new = label.copy()
        np.minimum.at(new, w, lo)
        np.minimum.at(new, f, lo)
        new = np.minimum(new, new[new])
        if (new == label).all():
            break
        label = new
    used = np.unique(f)
    score = np.bincount(label[used], minlength=label.size) * float(mass.sum() + 1)
    score = score + np.bincount(label[w], weights=mass[on], minlength=label.size)
    out = np.zeros(on.size, bool)
    out[np.flatnonzero(on)[label[w] == np.argmax(score)]] = True
    return out


def _retained(worker, firm, deletion):
    """The rows of the leave-out connected set: worker and firm are dense ids of every row."""
    W, F = worker.max() + 1, firm.max() + 1
    pair, row_pair, rows = np.unique(worker * F + firm, return_inverse=True, return_counts=True)
    pw, pf = pair // F, pair % F
    mass = rows.astype(float)
    on = _largest(pw, pf, mass, np.ones(pair.size, bool), W, F)
    if deletion == 1:
        on &= np.bincount(pw[on], minlength=W)[pw] > 1
    while True:
        on = _largest(pw, pf, mass, on, W, F)
        few = np.bincount(pw[on], minlength=W) == 1 if deletion == 1 else \
            np.bincount(pw[on], weights=mass[on], minlength=W) == 1
        if few.any():
            on &= ~few[pw]
            continue
        at = np.flatnonzero(on)
        cut, bridges = _low_points(W + F, pw[at], W + pf[at])
        if cut[:W].any():
            on &= ~cut[:W][pw]
        elif deletion == 1 and bridges.size:
            on[at[bridges]] = False
        else:
            return on[row_pair]


_M32 = np.uint64(0xFFFFFFFF)
_LEVERAGE, _TARGET = 0x4C45564552414745, 0x0054415247455401  # domain tags of the two probe kinds


def _mul(a, b):
    """High and low words of the 128-bit products a * b, a an integer below 2^64, b an array."""
    a0, a1 = np.uint64(a & 0xFFFFFFFF), np.uint64(a >> 32)
    b0, b1 = b & _M32, b >> np.uint64(32)
    p00, p01, p10 = a0 * b0, a0 * b1, a1 * b0
    mid = (p00 >> np.uint64(32)) + (p01 & _M32) + (p10 & _M32)
    return a1 * b1 + (p01 >> np.uint64(32)) + (p10 >> np.uint64(32)) + (mid >> np.uint64(32)), np.uint64(a) * b


def _splitmix(x):
    m = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & m
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & m
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & m
    return x ^ (x >> 31)


def _atoms(seed, tag, probes, entity, trials):
    """Rademacher sums of `trials` (at most 64) draws per entity and probe: Philox4x64-10 on the counter
    (entity, probe / 4, 0, tag), lane probe % 4."""
    m = (1 << 64) - 1
    blocks = (probes + 3) // 4
    shape = (entity.size, blocks)
    c = [np.broadcast_to(entity.astype(np.uint64)[:, None], shape).copy(),
         np.broadcast_to(np.arange(blocks, dtype=np.uint64), shape).copy(),
         np.zeros(shape, np.uint64), np.full(shape, tag, np.uint64)]
    k0, k1 = _splitmix(seed), _splitmix(seed ^ 0xD1B54A32D192ED03)
    for r in range(10):
        h0, l0 = _mul(0xD2B74407B1CE6E93, c[0])
        h1, l1 = _mul(0xCA5A826395121157, c[2])
        c = [h1 ^ c[1] ^ np.uint64(k0), l1, h0 ^ c[3] ^ np.uint64(k1), l0]
        k0, k1 = (k0 + 0x9E3779B97F4A7C15) & m, (k1 + 0xBB67AE8584CAA73B) & m
    keep = (np.uint64(1) << trials.astype(np.uint64)) - np.uint64(1)
    bits = np.stack([x & keep[:, None] for x in c], axis=2).reshape(entity.size, 4 * blocks)[:, :probes]
    return 2.0 * np.bitwise_count(bits) - trials[:, None]


class _Model:
    """The worker-firm least-squares model of a retained sample, solved by a dense factor of its firm block."""

    def __init__(self, worker, firm, outcome, controls):
        w = np.unique(worker, return_inverse=True)[1]
        f = np.unique(firm, return_inverse=True)[1]
        self.W, self.F = int(w.max()) + 1, int(f.max()) + 1
        cell, row_cell, n = np.unique(w * self.F + f, return_inverse=True, return_counts=True)
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.row_cell, self.count = self.t(row_cell), self.t(n.astype(float))
        self.cw, self.cf = self.t(cell // self.F), self.t(cell % self.F)
        self.y = self.t(outcome)
        self.Q = self.t(np.stack(controls, axis=1)) if len(controls) else self.y.new_zeros(self.y.numel(), 0)
        self.n = n
        self.dw = self.y.new_zeros(self.W).index_add_(0, self.cw, self.count)
        A = self.y.new_zeros(self.W, self.F)
        A[self.cw, self.cf] = self.count
        df = A.sum(0)
        L = torch.diag(df) - A.T @ (A / self.dw[:, None])
        self.factor = torch.linalg.cholesky(L[:-1, :-1])  # the last firm's effect is zero
        self.A = A

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def cells(self, per_row):
        return per_row.new_zeros(self.count.numel(), *per_row.shape[1:]).index_add_(0, self.row_cell, per_row)

    def solve(self, bw, bf):
        """Worker and firm effects of the right-hand sides (columns)."""
        b = bf - self.A.T @ (bw / self.dw[:, None])
        psi = torch.zeros_like(bf)
        psi[:-1] = torch.cholesky_solve(b[:-1], self.factor)
        return (bw - self.A @ psi) / self.dw[:, None], psi

    def fit(self, per_cell):
        """Cell predictions of the regressions on per-cell sums, and their effects."""
        k = per_cell.shape[1]
        a, p = self.solve(per_cell.new_zeros(self.W, k).index_add_(0, self.cw, per_cell),
                          per_cell.new_zeros(self.F, k).index_add_(0, self.cf, per_cell))
        return a[self.cw] + p[self.cf], a, p

    def plugin(self, a, p):
        t = self.count / self.count.sum()
        x, z = a[self.cw], p[self.cf]
        x, z = x - (t * x).sum(), z - (t * z).sum()
        return torch.stack([(t * x * x).sum(), (t * z * z).sum(), (t * x * z).sum(), (t * (x + z) ** 2).sum()])


def _finite(m, probes):
    """Projection and residual shares, bias and variance of the finite projection from five moment sums."""
    proj, res = m[0] / (m[0] + m[1]), m[1] / (m[0] + m[1])
    p4, r4, mix = m[2] / probes, m[3] / probes, m[4] / probes
    bias = (res * p4 - proj * r4 + (res - proj) * mix) / probes
    var = (res * res * p4 + proj * proj * r4 - 2 * proj * res * mix) / probes
    return proj, res, bias, var.clamp(min=0)


def _jla(case, panel, keep, seed):
    g = _Model(panel.worker[keep], panel.firm[keep], panel.outcome[keep], [c[keep] for c in panel.controls])
    P, y, Q, rc, n = case["probes"], g.y, g.Q, g.row_cell, g.count
    q, observation = Q.shape[1], case["deletion"] == 2
    before = np.cumsum(g.n) - g.n
    entity = (before + 1).astype(np.uint64)  # of a match or a target stratum: the first rank of its rows
    # the fit, jointly with the controls
    H, aH, pH = g.fit(g.cells(Q))
    R = Q - H[rc]
    S = torch.linalg.inv(R.T @ R)
    beta = S @ (R.T @ y)
    _, ay, py = g.fit(g.cells(y[:, None]))
    a, p = ay[:, 0] - aH @ beta, py[:, 0] - pH @ beta
    resid = y - (a[g.cw] + p[g.cf])[rc] - Q @ beta
    plugin = g.plugin(a, p)
    # leverages
    if observation:
        rank = np.empty(y.numel(), np.int64)
        rank[np.lexsort((panel.outcome[keep], rc.cpu().numpy()))] = np.arange(1, y.numel() + 1)
        atoms = g.t(_atoms(seed, _LEVERAGE, P, rank, np.ones(rank.size, np.int64)))
        u = g.fit(g.cells(atoms))[0][rc]
        zero = torch.zeros_like(y)
        first, third = (atoms * u).sum(1), (atoms * u ** 3).sum(1)
        f2, f4 = (u ** 2).sum(1), (u ** 4).sum(1)
        acc = torch.cat([torch.stack([f2, zero, f4, zero], 1).reshape(-1),
                         torch.stack([first, zero, third, zero], 1).reshape(-1)])
        proj, res, bias, var = _finite([f2, P + f2 - 2 * first, f4, P + 6 * f2 + f4 - 4 * first - 4 * third,
                                        f2 + f4 - 2 * third], P)
        t = res - ((R @ S) * R).sum(1)
        deleted = resid * (1 / t + bias / t ** 2 - var / t ** 3)
    else:
        atoms = g.t(_atoms(seed, _LEVERAGE, P, entity, g.n))
        u = n.sqrt()[:, None] * g.fit(atoms)[0]
        m = atoms / n.sqrt()[:, None] - u
        mom = [(u ** 2).sum(1), (m ** 2).sum(1), (u ** 4).sum(1), (m ** 4).sum(1), (u ** 2 * m ** 2).sum(1)]
        acc = torch.stack(mom, 1).reshape(-1)
        proj, res, bias, var = _finite(mom, P)
        if q == 0:
            deleted = g.cells(resid[:, None])[:, 0] * (1 / res + bias / res ** 2 - var / res ** 3)
        else:  # per match block: I - (share of the match mean) - (control leverage)
            order = torch.argsort(rc, stable=True)
            start = g.t(before)
            deleted = torch.zeros_like(y)
            for k in np.unique(g.n).tolist():
                at = torch.nonzero(n == k)[:, 0]
                rows = order[start[at][:, None] + torch.arange(k, device=g.dev)]
                Rb, c = R[rows], torch.full((at.numel(), k, 1), k ** -0.5, dtype=y.dtype, device=g.dev)
                M = torch.eye(k, dtype=y.dtype, device=g.dev) - proj[at][:, None, None] * c @ c.mT - Rb @ S @ Rb.mT
                x = torch.linalg.solve(M, torch.cat([resid[rows][:, :, None], c], 2))
                x0, x1 = x[:, :, 0], x[:, :, 1]
                ct, ci = (c[:, :, 0] * x0).sum(1, True), (c[:, :, 0] * x1).sum(1, True)
                deleted[rows] = x0 + bias[at][:, None] * x1 * ct - var[at][:, None] * x1 * ci * ct
    # target probes: a worker-side and a firm-side solve each
    d = g.t(_atoms(seed, _TARGET, P, entity, g.n)) / n.sum().sqrt()
    d = d - (n / n.sum())[:, None] * d.sum(0)
    sides = []
    for side in (0, 1):
        bw, bf = d.new_zeros(g.W, P), d.new_zeros(g.F, P)
        (bw if side == 0 else bf).index_add_(0, (g.cw, g.cf)[side], d)
        x, z = g.solve(bw, bf)
        v = (x[g.cw] + z[g.cf])
        b = -S @ (Q.T @ v[rc])
        sides.append((v, b))
    sides.append((sides[0][0] + sides[1][0], sides[0][1] + sides[1][1]))
    if q == 0 and not observation:
        om = g.cells(y[:, None])[:, 0] * deleted
        worker, firm, cov = [(om[:, None] * s * r).sum(0) for s, r in
                             ((sides[0][0], sides[0][0]), (sides[1][0], sides[1][0]), (sides[0][0], sides[1][0]))]
    else:
        quad = []
        for v, b in sides:
            pred = v[rc] + R @ b
            if observation:
                quad.append(((y * deleted)[:, None] * pred ** 2).sum(0))
            else:
                quad.append((g.cells(y[:, None] * pred) * g.cells(deleted[:, None] * pred)).sum(0))
        worker, firm, cov = quad[0], quad[1], 0.5 * (quad[2] - quad[0] - quad[1])
    draws = torch.stack([worker, firm, cov, worker + firm + 2 * cov], 1)
    corr = draws.mean(0)
    mcse = (((draws - corr) ** 2).sum(0) / (P * (P - 1.0))).sqrt()
    host = {k: v.cpu().numpy() for k, v in dict(draws=draws, plugin=plugin, correction=corr, corrected=plugin - corr,
                                                numerical_mcse=mcse).items()}
    return dict(host, accumulators=acc)


def _leverages(panel, keep):
    g = _Model(panel.worker[keep], panel.firm[keep], panel.outcome[keep], [])
    n, y = g.count, g.cells(g.y[:, None])[:, 0]
    t = n / n.sum()
    fit, a, p = g.fit(y[:, None])
    resid, corr = y - n * fit[:, 0], torch.zeros(4, dtype=y.dtype, device=g.dev)
    sw = t.new_zeros(g.W).index_add_(0, g.cw, t)[:, None]
    sf = t.new_zeros(g.F).index_add_(0, g.cf, t)[:, None]
    for at in torch.arange(n.numel(), device=g.dev).split(512):
        one = torch.arange(at.numel(), device=g.dev)
        bw, bf = y.new_zeros(g.W, at.numel()), y.new_zeros(g.F, at.numel())
        bw[g.cw[at], one] = 1.0
        bf[g.cf[at], one] = 1.0
        x, z = g.solve(bw, bf)
        h = x[g.cw[at], one] + z[g.cf[at], one]
        om = y[at] * resid[at] / (1 - n[at] * h)
        ww = (sw * x * x).sum(0) - (sw * x).sum(0) ** 2
        ff = (sf * z * z).sum(0) - (sf * z).sum(0) ** 2
        cv = (t[:, None] * x[g.cw] * z[g.cf]).sum(0) - (sw * x).sum(0) * (sf * z).sum(0)
        corr += torch.stack([(om * ww).sum(), (om * ff).sum(), (om * cv).sum(), (om * (ww + ff + 2 * cv)).sum()])
    plugin = g.plugin(a[:, 0], p[:, 0])
    host = lambda x: x.cpu().numpy()  # noqa: E731
    return {"plugin": host(plugin), "correction": host(corr), "corrected": host(plugin - corr),
            "numerical_mcse": None}


def _gradient(case, seed):
    """Loss and gradient of the network by reverse-mode differentiation in 64 bits; its weights are BF16."""
    with_trainer = prepare(case, seed)["trainer"]
    d, params = with_trainer.dump(0), with_trainer.params
    with_trainer.close()
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev).double()  # noqa: E731
    n, P, diag = d["n"], d["pairs"], t(d["diag"])
    row = torch.from_numpy(np.repeat(np.arange(n), np.diff(d["ptr"].astype(np.int64)))).to(dev)
    col = torch.from_numpy(d["col"].astype(np.int64)).to(dev)
    A = torch.sparse_coo_tensor(torch.stack([row, col]), t(d["val"]), (n, n)).coalesce()
    x = t(params).requires_grad_(True)
    w = x + (torch.from_numpy(params).bfloat16().double().to(dev) - x.detach())
    h, o = t(d["X"]), 0
    for layer in range(4):
        i = h.shape[1]
        ws, wn = w[o:o + 64 * i].reshape(i, 64), w[o + 64 * i:o + 128 * i].reshape(i, 64)
        h = torch.relu(h @ ws + (torch.sparse.mm(A, h) / diag[:, None]) @ wn + x[o + 128 * i:o + 128 * i + 64])
        o += 128 * i + 64
    c = h @ w[o:o + 128].reshape(64, 2) + x[o + 128:o + 130]
    s = torch.nn.functional.softplus(c[:, 1])
    a = s * s + 0.01 + torch.nn.functional.softplus(c[:, 0])
    y0, energy = t(d["Y"]).reshape(n, P), t(d["ELE"])
    z = a[:, None] * y0 + (s / diag)[:, None] * torch.sparse.mm(A, s[:, None] * y0)
    top = (z * diag[:, None] * y0).sum(0)
    bottom = (z * (diag[:, None] * z - torch.sparse.mm(A, z))).sum(0)
    ok = (energy > 0) & (bottom > 0)
    loss = torch.where(ok, 1 - top ** 2 / torch.where(ok, energy * bottom, torch.ones_like(energy)), 0.0).sum() / P
    loss.backward()
    return {"loss": np.float64(loss.item()), "gradient": x.grad.cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "train":
        return _gradient(case, seed)
    if case["workers"] > 25_000:  # the search for the connected set and the dense factor take too long
        return None
    panel = _panel(case, 20261203 if case["kind"] == "shard" else seed)
    worker, firm = (np.unique(x, return_inverse=True)[1] for x in (panel.worker, panel.firm))
    keep = _retained(worker, firm, case["deletion"])
    if case["kind"] == "exact":
        return dict(_leverages(panel, keep), retained=keep.astype(np.uint8))
    got = _jla(case, panel, keep, 1 + seed)
    if case["kind"] == "shard":
        return got
    del got["accumulators"], got["draws"]
    if case["numerical"]:
        got.update(status=None, covariance=None, mcse=None)
    return dict(got, retained=keep.astype(np.uint8))
