"""Timed cases of the engine, each through a public entry point of the package.

A case is a dict of plain values.  `path` says which entry point it takes:

  advance    PdhgBackend, one check interval of the iteration seam: start points
             up, INTERVAL PDHG trials, current and averaged points back.  What
             the reference's driver does between two candidate checks, and
             where nearly all time of a solve goes.
  batch      BatchEngine.step(1), one check interval (100 trials, candidate
             evaluation, restarts) of a resident batch of uneven LPs and QPs.
             What the service runs in a loop.
  batch_call solve_batch, a whole call on a few small models.
  solve      solver.solve, a whole call: presolve, scaling, iterations, checks
             and the host certificate, on an iteration budget.
  newton     linear_solve, one Newton system of the barrier method.
  propagate  propagate_bounds, one GPU presolve / branch-and-bound node call.

Every input comes from the seed alone.  Matrices are drawn on the GPU and handed
over as host CSR arrays, which is what the entry points take.
"""
from __future__ import annotations

import math
import types

import numpy as np
import torch

from niryukti_b200 import batch, engine, solver

CHECK = 100    # the drivers' default check interval, in trials
# Trials of an `advance` pass.  Adaptive steps carry last-bit differences between
# two correct orders of summation forward, about tenfold every eight trials; at 40
# the points still agree to twelve digits.
INTERVAL = 40
HI = 10.0      # upper bound of a boxed column


def listed():
    return [
        # a small planning LP, 2,000 x 5,000 with 5 entries per column: every
        # vector fits on chip, so the time of a trial is launches and latency
        dict(name="lp_small", path="advance", pattern="column", m=2000, n=5000, per=5,
             method="adaptive", precision="fp64"),
        # an ordinary LP of odd sizes whose matrices stay in L2
        dict(name="lp_medium", path="advance", pattern="column", m=30011, n=60037, per=6,
             method="adaptive", precision="fp64"),
        # the 20M-entry LP with power-law rows: the largest single model
        dict(name="lp_power_law", path="advance", pattern="power", m=1_000_000, n=2_000_000,
             per=10, method="adaptive", precision="fp64"),
        # the same family, ragged and smaller, on FP32 values
        dict(name="lp_power_law_mixed", path="advance", pattern="power", m=250_007, n=500_009,
             per=10, method="adaptive", precision="mixed"),
        # block-angular planning LP: blocks joined by long linking rows
        dict(name="lp_block_angular", path="advance", pattern="block", m=60_000, n=120_000,
             per=6, blocks=6, linking=1500, method="adaptive", precision="fp64"),
        # a convex QP with a sparse Q = D + L L^T (fixed steps)
        dict(name="qp_sparse", path="advance", pattern="column", m=10_000, n=20_000, per=6,
             qp=True, method="fixed", precision="fp64"),
        # Halpern-anchored fixed steps, the reference's other first-order form
        dict(name="lp_halpern", path="advance", pattern="column", m=50_021, n=120_011, per=5,
             method="halpern", precision="fp64"),
        # a resident batch of 96 uneven LPs and QPs, as bench and service run it
        dict(name="batch_96", path="batch", count=96, m_lo=500, m_hi=50_000, precision="fp64"),
        # a whole batched call on two dozen small models, on the service's precision
        dict(name="batch_call_24", path="batch_call", count=24, m_lo=500, m_hi=3000, checks=10,
             precision="mixed"),
        # a whole solve of the small LP on a budget of 2,000 iterations
        dict(name="solve_small", path="solve", pattern="column", m=2000, n=5000, per=5,
             checks=20, precision="fp64"),
        # a barrier Newton system (saddle point of 24,000 unknowns)
        dict(name="newton_saddle", path="newton", m=8000, n=16_000, per=5),
        # five rounds of bound propagation over a half-integer model
        dict(name="propagate", path="propagate", m=20_000, n=40_000, per=8, passes=5),
    ]


def _size(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm, odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["advance"] * 6 + ["batch", "batch_call", "solve", "newton", "propagate"])
    if path == "advance":
        pattern = rng.choice(["column", "column", "column", "power", "power", "block"])
        method = rng.choice(["adaptive"] * 4 + ["fixed", "halpern"])
        precision = rng.choice(["fp64", "fp64", "fp64", "mixed"])
        if pattern == "column":
            m = _size(rng, 500, 200_000)
            n = int(m * rng.uniform(1.5, 3.0))
            qp = rng.random() < 0.25
            if qp:
                m, n = max(500, m // 4), max(1000, n // 4)
            return dict(path=path, pattern=pattern, m=m, n=n, per=rng.randint(4, 8), qp=qp,
                        method="fixed" if qp else method, precision="fp64" if qp else precision)
        if pattern == "power":
            m = _size(rng, 5000, 700_000)
            return dict(path=path, pattern=pattern, m=m, n=int(m * rng.uniform(1.5, 2.2)),
                        per=rng.randint(7, 10), method=method, precision=precision)
        blocks, rows = rng.randint(2, 6), _size(rng, 1000, 10_000)
        return dict(path=path, pattern=pattern, m=blocks * rows, n=2 * blocks * rows, per=6,
                    blocks=blocks, linking=_size(rng, 100, 1500), method=method,
                    precision=precision)
    if path == "batch":
        return dict(path=path, count=_size(rng, 8, 128), m_lo=500,
                    m_hi=_size(rng, 2000, 30_000), precision=rng.choice(["fp64", "fp64", "mixed"]))
    if path == "batch_call":
        return dict(path=path, count=rng.randint(4, 24), m_lo=500, m_hi=_size(rng, 1000, 4000),
                    checks=rng.randint(4, 12), precision=rng.choice(["fp64", "mixed"]))
    if path == "solve":
        m = _size(rng, 500, 20_000)
        return dict(path=path, pattern="column", m=m, n=int(m * rng.uniform(1.5, 3.0)),
                    per=rng.randint(4, 8), checks=rng.randint(5, 20), precision="fp64")
    m = _size(rng, 500, 30_000)
    if path == "newton":
        return dict(path=path, m=m, n=int(m * rng.uniform(1.2, 2.5)), per=rng.randint(3, 6))
    return dict(path=path, m=m, n=int(m * rng.uniform(1.5, 2.5)), per=rng.randint(4, 10),
                passes=rng.randint(2, 8))


# ------------------------------------------------------------------ models
class _Draw:
    """Random numbers of one seed, on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, device="cuda",
                                           dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def integers(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device="cuda")


def _row_sums(ptr, weighted):
    out = np.zeros(len(ptr) - 1)
    full = np.diff(ptr) > 0
    if weighted.size:
        out[full] = np.add.reduceat(weighted, ptr[:-1][full])
    return out


def _csr(keys, rows, cols):
    """Host ptr and idx of the distinct keys (row * cols + column)."""
    keys = torch.unique(keys)
    r = keys // cols
    ptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(r, minlength=rows), 0)
    return ptr.cpu().numpy(), (keys - r * cols).cpu().numpy(), r


def _power_lengths(d, m, mean, lo=2, hi=5000):
    """m row lengths on [lo, hi] from a power law of that mean."""
    lens = torch.arange(lo, hi + 1, dtype=torch.float64)
    a, b = 0.5, 4.0
    for _ in range(60):
        mid = 0.5 * (a + b)
        w = lens ** -mid
        if float((lens * w).sum() / w.sum()) > mean:
            a = mid
        else:
            b = mid
    cdf = torch.cumsum(lens ** -b, 0)
    cdf = (cdf / cdf[-1]).cuda()
    return lo + torch.searchsorted(cdf, d.uniform(0, 1, m)).clamp(max=hi - lo)


def _model(case, seed):
    """An LP or convex QP, feasible at a point of its own."""
    d = _Draw(seed)
    m, n, pattern = case["m"], case["n"], case.get("pattern", "column")
    if pattern == "column":
        cols = torch.arange(n, device="cuda").repeat_interleave(case["per"])
        ptr, idx, r = _csr(d.integers(m, cols.numel()) * n + cols, m, n)
        val = d.normal(len(idx))
    elif pattern == "power":
        lens = _power_lengths(d, m, case["per"] * n / m)
        rows = torch.arange(m, device="cuda").repeat_interleave(lens)
        ptr, idx, r = _csr(rows * n + d.integers(n, rows.numel()), m, n)
        factor = torch.exp(d.uniform(math.log(1e-2), math.log(1e2), m))
        val = d.normal(len(idx)) * factor[r]
    else:
        block_rows, block_cols = m // case["blocks"], n // case["blocks"]
        cols = torch.arange(n, device="cuda").repeat_interleave(case["per"])
        own = (cols // block_cols) * block_rows + d.integers(block_rows, cols.numel())
        link = case["linking"]
        joined = torch.arange(m, m + link, device="cuda").repeat_interleave(n // 20)
        m = m + link
        ptr, idx, r = _csr(torch.cat([own * n + cols, joined * n + d.integers(n, joined.numel())]),
                           m, n)
        val = d.uniform(0.1, 2.0, len(idx))
        val = torch.where(d.uniform(0, 1, len(idx)) < 0.3, -val, val)
    val = val.cpu().numpy()
    x0 = d.uniform(0, HI if pattern != "power" else 5.0, n).cpu().numpy()
    ax = _row_sums(ptr, val * x0[idx])
    rl, ru = ax.copy(), ax.copy()
    lb, ub = np.zeros(n), np.full(n, HI if pattern != "block" else 2 * HI)
    if pattern == "power":      # half the rows <=, a tenth of the columns free
        rl[m // 2:] = -np.inf
        ru[m // 2:] += d.uniform(0, 1, m - m // 2).cpu().numpy()
        free = d.uniform(0, 1, n).cpu().numpy() < 0.1
        lb[free], ub[free] = -np.inf, np.inf
    elif pattern == "block":    # the linking rows are <=
        rl[-case["linking"]:] = -np.inf
        ru[-case["linking"]:] += 1.0
    c = d.normal(n).cpu().numpy()
    out = types.SimpleNamespace(m=m, n=n, ptr=ptr, idx=idx, val=val, c=c, q=np.zeros(n), lb=lb,
                                ub=ub, rl=rl, ru=ru, qptr=None, qidx=None, qval=None, qnnz=0,
                                offset=0.0)
    if case.get("qp"):          # Q = D + L L^T, D on the diagonal, L of four sparse columns
        s = min(n, int(math.ceil(math.sqrt(n))))
        pairs, prods = [], []
        for _ in range(4):
            at = torch.randperm(n, generator=d.g, device="cuda")[:s]
            v = 0.1 * d.normal(s)
            pairs.append((at[:, None] * n + at[None, :]).reshape(-1))
            prods.append((v[:, None] * v[None, :]).reshape(-1))
        keys, prods = torch.cat(pairs).cpu().numpy(), torch.cat(prods).cpu().numpy()
        distinct, inverse = np.unique(keys, return_inverse=True)
        out.qval = np.bincount(inverse, weights=prods, minlength=distinct.size)
        out.qidx = distinct % n
        out.qptr = np.zeros(n + 1, dtype=np.int64)
        np.cumsum(np.bincount(distinct // n, minlength=n), out=out.qptr[1:])
        out.qnnz = int(distinct.size)
        out.q = d.uniform(0.1, 1.0, n).cpu().numpy()
    return out


def _propagation_model(case, seed):
    """Covering and packing rows with positive coefficients over wide boxes, every
    second column integer: the activity bounds imply most upper bounds."""
    out = _model(case, seed)
    d = _Draw(seed + 104729)
    n, m = case["n"], case["m"]
    out.val = np.abs(out.val) + 0.1
    out.integer = (np.arange(n) % 2 == 0).astype(np.int32)
    x0 = d.uniform(0, HI, n).cpu().numpy()
    x0[out.integer == 1] = np.floor(x0[out.integer == 1])
    ax = _row_sums(out.ptr, out.val * x0[out.idx])
    slack = d.uniform(0, 1, m).cpu().numpy()
    out.ru = ax + slack
    out.rl = np.where(np.arange(m) % 3 == 0, -np.inf, ax - slack)
    out.ub = np.full(n, 100 * HI)
    return out


def _batch_models(case, seed):
    """Uneven LPs with every fifth a QP: m log-uniform, n = 2m, 4 to 8 entries per column."""
    spread = math.log(case["m_hi"] / case["m_lo"])
    got = []
    for k in range(case["count"]):
        m = int(case["m_lo"] * math.exp(spread * ((k * 0.618033988749895) % 1.0)))
        got.append(_model(dict(m=m, n=2 * m, per=4 + k % 5, qp=k % 5 == 4), 1000 * seed + k))
    return got


def _steps(model):
    """The driver's first step sizes: 0.9 / sqrt(|A|_inf |A|_1) and |c| / |b| as the weight."""
    a = np.abs(model.val)
    norm = math.sqrt(_row_sums(model.ptr, a).max()) * math.sqrt(
        np.bincount(model.idx, weights=a, minlength=model.n).max())
    b = np.clip(0.0, model.rl, model.ru)
    weight = min(1e4, max(1e-4, math.sqrt(float(model.c @ model.c) / float(b @ b))))
    return 0.9 / norm / weight, 0.9 / norm * weight


def _start(model, seed):
    """A start point inside the bounds and a small dual one, as after a restart."""
    d = _Draw(seed + 7919)
    x = np.clip(d.uniform(0, 5.0, model.n).cpu().numpy(), model.lb, model.ub)
    y = 0.1 * d.normal(model.m).cpu().numpy()
    y[np.isinf(model.rl)] = np.abs(y[np.isinf(model.rl)])
    return x, y


def _pinned(a):
    t = torch.empty(a.shape[0], dtype=torch.float64, pin_memory=True)
    t.copy_(torch.from_numpy(a))
    return t.numpy()


def _newton_system(case, seed):
    """Saddle point K = [H A^T; A -R] of one barrier iteration: H and R diagonal."""
    d = _Draw(seed)
    m, n = case["m"], case["n"]
    cols = torch.arange(n, device="cuda").repeat_interleave(case["per"])
    keys = torch.unique(d.integers(m, cols.numel()) * n + cols)
    r, j = keys // n, keys % n
    a = 0.3 * d.normal(keys.numel())
    h, reg = d.uniform(1.0, 4.0, n), d.uniform(1.0, 2.0, m)
    diag = torch.arange(n + m, device="cuda")
    rows = torch.cat([diag, j, n + r])
    cols = torch.cat([diag, n + r, j])
    vals = torch.cat([h, -reg, a, a])
    order = torch.argsort(rows * (n + m) + cols)
    ptr = np.zeros(n + m + 1, dtype=np.int64)
    np.cumsum(torch.bincount(rows, minlength=n + m).cpu().numpy(), out=ptr[1:])
    return dict(ptr=ptr, idx=cols[order].cpu().numpy(), val=vals[order].cpu().numpy(),
                rhs=d.normal(n + m).cpu().numpy(), h=h, reg=reg, a=(r, j, a))


# ------------------------------------------------------------------ the cases' hooks
def prepare(case, seed):
    path = case["path"]
    s = types.SimpleNamespace(case=case)
    if path == "advance":
        model = _model(case, seed)
        s.x, s.y = (_pinned(v) for v in _start(model, seed))
        s.tau, s.sigma = _steps(model)
        s.out = tuple(_pinned(np.zeros(k)) for k in (model.n, model.m, model.n, model.m))
        s.backend = engine.PdhgBackend(model, s.x, s.y, adaptive=case["method"] == "adaptive",
                                       halpern=case["method"] == "halpern", graphs=True,
                                       precision=case["precision"])
    elif path == "batch":
        # a tolerance nothing reaches: the batch stays full, as admission keeps it
        s.engine = batch.BatchEngine(tol=1e-13, iteration_limit=10**9, time_limit=1e9,
                                     matrix_precision=case["precision"])
        for k, model in enumerate(_batch_models(case, seed)):
            if not s.engine.admit(s.engine.prepare(model), k):
                raise MemoryError("the batch does not fit")
    elif path == "batch_call":
        s.models = _batch_models(case, seed)
    elif path == "solve":
        s.model = _model(case, seed)
    elif path == "newton":
        s.system = _newton_system(case, seed)
    else:
        s.model = _propagation_model(case, seed)
        s.integer = s.model.integer
    return s


def run(s):
    case = s.case
    path = case["path"]
    if path == "advance":
        s.backend.reset(s.x, s.y)
        s.backend.advance(INTERVAL, s.tau, s.sigma)
        return s.backend.candidates(out=s.out)
    if path == "batch":
        s.engine.step(checks=1)
        got = [s.engine.progress(k) for k in range(case["count"])]
        return {key: np.array([p[key] for p in got]) for key in got[0]}
    if path == "batch_call":
        got = batch.solve_batch(s.models, iteration_limit=CHECK * case["checks"],
                                matrix_precision=case["precision"])
        return [(r["x"], r["y"]) for r in got]
    if path == "solve":
        r = solver.solve(s.model, iteration_limit=CHECK * case["checks"],
                         matrix_precision=case["precision"])
        return {"x": r["x"], "y": r["y"], "objective": r["objective"], "kkt": r["kkt"],
                "iterations": r["iterations"]}
    if path == "newton":
        k = s.system
        x, ok = engine.linear_solve(k["ptr"], k["idx"], k["val"], k["rhs"])
        return {"x": x, "converged": ok}
    ok, lb, ub = engine.propagate_bounds(s.model, s.integer, s.model.lb, s.model.ub,
                                         passes=case["passes"])
    return {"feasible": ok, "lb": lb, "ub": ub}


def work(case):
    """What a pass cannot do without: per trial, each matrix entry of A and of
    A^T (value and 32-bit index), the row offsets, and the iterates' vectors;
    host-side entry points: the arrays they are given and return."""
    path = case["path"]

    def trial(m, n, nnz, qnnz=0, value=8):
        return (2 * nnz + qnnz) * (value + 4) + 4 * (m + n) + 8 * (9 * n + 9 * m), \
            4 * nnz + 2 * qnnz + 20 * (m + n)

    def q_entries(n):
        return 4 * math.ceil(math.sqrt(n)) ** 2

    if path in ("batch", "batch_call"):
        spread = math.log(case["m_hi"] / case["m_lo"])
        total = [0.0, 0.0]
        for k in range(case["count"]):
            m = int(case["m_lo"] * math.exp(spread * ((k * 0.618033988749895) % 1.0)))
            b, f = trial(m, 2 * m, 2 * m * (4 + k % 5), q_entries(2 * m) if k % 5 == 4 else 0,
                         8 if case["precision"] == "fp64" else 4)
            total = [total[0] + b, total[1] + f]
        times = CHECK * case.get("checks", 1)
        return {"bytes": times * total[0], "flops": times * total[1]}
    m, n = case["m"], case["n"]
    nnz = n * case["per"]
    if path == "newton":  # about 30 iterations of two products and ten vector passes
        size = m + n
        return {"bytes": 30 * (2 * (2 * nnz + size) * 12 + 10 * 8 * size),
                "flops": 30 * (4 * (2 * nnz + size) + 20 * size)}
    if path == "propagate":
        return {"bytes": 16 * nnz + 8 * m + 16 * m + 20 * n + 16 * n,
                "flops": case["passes"] * 12 * nnz}
    if case["pattern"] == "block":
        nnz += case["linking"] * (n // 20)
        m += case["linking"]
    b, f = trial(m, n, nnz, q_entries(n) if case.get("qp") else 0,
                 8 if case["precision"] == "fp64" else 4)
    times = CHECK * case["checks"] if path == "solve" else INTERVAL
    return {"bytes": times * b, "flops": times * f}


# ------------------------------------------------------------------ plain FP64
def _sparse(ptr, idx, val, rows, cols):
    t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (ptr, idx, val)]
    return torch.sparse_csr_tensor(*t, size=(rows, cols), check_invariants=False)


def _exact_advance(case, seed):
    """The pass of `advance`, trial by trial, in plain torch."""
    p = _model(case, seed)
    tau0, sigma0 = _steps(p)
    x, y, c, q, lb, ub, rl, ru = (torch.from_numpy(v).cuda() for v in
                                  (*_start(p, seed), p.c, p.q, p.lb, p.ub, p.rl, p.ru))
    A = _sparse(p.ptr, p.idx, p.val, p.m, p.n)
    rows = np.repeat(np.arange(p.m), np.diff(p.ptr))
    order = np.lexsort((rows, p.idx))
    tptr = np.zeros(p.n + 1, dtype=np.int64)
    np.cumsum(np.bincount(p.idx, minlength=p.n), out=tptr[1:])
    At = _sparse(tptr, rows[order], p.val[order], p.n, p.m)
    Q = _sparse(p.qptr, p.qidx, p.qval, p.n, p.n) if p.qnnz else None
    if Q is not None:  # the step bound of a QP
        a = np.abs(p.val)
        norm = math.sqrt(_row_sums(p.ptr, a).max()) * math.sqrt(
            np.bincount(p.idx, weights=a, minlength=p.n).max())
        qnorm = float((_row_sums(p.qptr, np.abs(p.qval)) + np.abs(p.q)).max())
        safety = math.sqrt(tau0 * sigma0) * norm + tau0 * qnorm
        scale = min(1.0, 0.9 / safety)
        tau0, sigma0 = tau0 * scale, sigma0 * scale
    adaptive, halpern = case["method"] == "adaptive" and Q is None, case["method"] == "halpern"
    ax = A @ x
    anchor = x, y, ax
    xa, ya = torch.zeros_like(x), torch.zeros_like(y)
    factor, mass, accepted, epoch = 1.0, 0.0, 0, 0
    for _ in range(INTERVAL):
        tau, sigma = tau0 * factor, sigma0 * factor
        g = c + At @ y
        if Q is not None:
            t = x - tau * (g + (Q @ x + q * x))
        else:
            t = (x - tau * g) / (1 + tau * q)
        t = torch.minimum(torch.maximum(t, lb), ub)
        dx = t - x
        delta = A @ dx
        z = y + sigma * (ax + 2 * delta)
        u = (z - sigma * ru).clamp(min=0) + (z - sigma * rl).clamp(max=0)
        dy, axt = u - y, ax + delta
        energy = float(dx @ dx) / tau + float(dy @ dy) / sigma
        cross = abs(float(dy @ delta))
        limit = energy / (2 * cross) if cross > 0 else math.inf
        accept, used = not adaptive or limit >= 1, factor
        if adaptive:
            k = accepted + 2
            factor = used * min((1 - k ** -0.3) * limit, 1 + k ** -0.6)
        if not accept:
            continue
        mass += used
        accepted += 1
        if halpern:
            lam = 1 / (epoch + 2)
            epoch += 1
            xa, ya = t, u
            x, y, ax = (lam * a + (1 - lam) * v for a, v in zip(anchor, (t, u, axt)))
        else:
            x, y, ax = t, u, axt
            xa, ya = xa + (x - xa) * (used / mass), ya + (y - ya) * (used / mass)
    return tuple(v.cpu().numpy() for v in (x, y, xa, ya))


def _exact_newton(case, seed):
    """x of the saddle point by conjugate gradients on (R + A H^-1 A^T)."""
    k = _newton_system(case, seed)
    m, n = case["m"], case["n"]
    (r, j, a), h, reg = k["a"], k["h"], k["reg"]
    A = torch.sparse_coo_tensor(torch.stack([r, j]), a, (m, n)).to_sparse_csr()
    At = torch.sparse_coo_tensor(torch.stack([j, r]), a, (n, m)).to_sparse_csr()
    f, g = (torch.from_numpy(v).cuda() for v in (k["rhs"][:n], k["rhs"][n:]))
    b = A @ (f / h) - g
    y = torch.zeros_like(b)
    for _ in range(3):  # restarted on the true residual
        res = b - (reg * y + A @ ((At @ y) / h))
        p, rr = res.clone(), float(res @ res)
        for _ in range(200):
            if rr < 1e-34 * float(b @ b):
                break
            w = reg * p + A @ ((At @ p) / h)
            alpha = rr / float(p @ w)
            y = y + alpha * p
            res = res - alpha * w
            rr, before = float(res @ res), rr
            p = res + (rr / before) * p
    x = (f - At @ y) / h
    return {"x": torch.cat([x, y]).cpu().numpy(), "converged": None}


def exact(case, seed):
    """FP64 values of `run` for a fresh state.  None where a pass goes through
    presolve, scaling and the restart driver (batch, batch_call, solve) or is
    defined by its directed rounding (propagate)."""
    if case["path"] == "advance":
        return _exact_advance(case, seed)
    if case["path"] == "newton":
        return _exact_newton(case, seed)
    return None
