"""The B200 engine against the oracle, step by step (the reference's own parity
contract: tests/test_research.cpp:34-64,740-761,839-907; 1e-11 relative).

Each case runs the engine through its C ABI (niryukti_b200.engine) beside the
C oracle on the same inputs.  Where the engine's SpMV sums a row in a different
order than the CPU, agreement is to rounding (tolerances written per test)."""
import json
import math

import numpy as np
import pytest

from niryukti_b200 import synth
from tests.conftest import load_golden
from tests.test_oracle import halpern_expected, sparse_qp_model, tiny

pytestmark = pytest.mark.gpu


def step_sizes(model):
    """tau, sigma as solve_continuous starts them (src/solver.cpp:299-333)."""
    import bench
    return bench.step_sizes(model)


def near(a, b, tol=1e-11):
    a, b = np.asarray(a, dtype=float), np.asarray(b, dtype=float)
    err = np.abs(a - b) / (1 + np.abs(b))
    assert np.all(err <= tol), f"max rel err {err.max():.3e} > {tol}"


def advance_to(g, target, tau, sigma, done=0):
    """Run single trials until `target` accepted steps.  The CPU backend counts
    accepted iterations (retrying each up to 40 times, src/cpu.cpp:103-221); the
    CUDA backend counts trials (src/cuda.cu:849-866), so adaptive trajectories
    line up at equal accepted counts."""
    for _ in range(40 * max(1, target - done) + 40):
        if done >= target:
            return done
        done += g.advance(1, tau, sigma)
    raise AssertionError(f"no progress to {target} accepted steps")


def test_acceptance_parity(gpu, oracle):
    # tests/test_research.cpp:34-64
    m = tiny(1, 1, [(0, 0, 1.0)])
    m.c[:] = -1
    m.rl[:] = m.ru[:] = 3
    cpu = oracle.model(m).backend(np.zeros(1), np.zeros(1), adaptive=True)
    assert cpu.advance(1, 2, 2) == 1
    g = gpu.PdhgBackend(m, adaptive=True)
    accepted = 0
    for _ in range(40):
        if accepted:
            break
        accepted += g.advance(1, 2, 2)
    assert accepted == 1
    assert g.rejected_steps() == cpu.rejected_steps()
    for u, w in zip(g.candidates(), cpu.candidates()):
        near(u, w)


def test_halpern_scalar_recurrence(gpu):
    m = tiny(1, 1, [(0, 0, 1.0)])
    m.lb[:] = -math.inf
    m.ub[:] = math.inf
    m.rl[:] = m.ru[:] = 1
    g = gpu.PdhgBackend(m, halpern=True)
    for ex, ey, tx, ty in halpern_expected():
        g.advance(1, .5, .5)
        x, y, rx, ry = g.candidates()
        near(x[0], ex)
        near(y[0], ey)
        near(rx[0], tx)
        near(ry[0], ty)
    g.reset(np.array([2.0]), np.array([3.0]))
    g.advance(1, .5, .5)
    x, y, _, _ = g.candidates()
    near(x[0], 1.25)
    near(y[0], 2.5)


@pytest.mark.parametrize("reflection", [0.0, 1.0])
@pytest.mark.parametrize("graphs", [False, True])
def test_anchored_parity(gpu, oracle, reflection, graphs):
    # tests/test_research.cpp:864-891
    m = tiny(2, 2, [(0, 0, 1.0), (0, 1, 2.0), (1, 0, -1.0), (1, 1, 1.0)])
    m.c = np.array([1.0, -2.0])
    m.rl = np.array([-1.0, -2.0])
    m.ru = np.array([3.0, 2.0])
    cpu = oracle.model(m).backend(np.zeros(2), np.zeros(2), halpern=True, reflection=reflection)
    g = gpu.PdhgBackend(m, halpern=True, reflection=reflection, graphs=graphs, indices="32")
    for k in range(30):
        assert cpu.advance(1, .1, .1) == g.advance(1, .1, .1)
        c = cpu.candidates()
        d = g.candidates()
        for u, w in zip(d, c):
            near(u, w)
        if k == 14:
            cpu.reset(c[0], c[1])
            g.reset(d[0], d[1])


@pytest.mark.parametrize("width", ["32", "64"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_width_precision_parity(gpu, oracle, width, precision):
    # tests/test_research.cpp:892-907
    m = tiny(2, 2, [(0, 0, 1.0), (0, 1, 2.0), (1, 0, -1.0), (1, 1, 1.0)])
    m.c = np.array([1.0, -2.0])
    m.rl = np.array([-1.0, -2.0])
    m.ru = np.array([3.0, 2.0])
    cpu = oracle.model(m).backend(np.zeros(2), np.zeros(2))
    g = gpu.PdhgBackend(m, graphs=True, indices=width, precision=precision)
    cpu.advance(30, .1, .1)
    g.advance(30, .1, .1)
    mon = g.monitor()
    c, d = cpu.candidates(), g.candidates()
    near(d[0], c[0])
    near(d[1], c[1])
    # the KKT proxy against the FP64 host evaluation of the reference's formula
    # on the engine's own current and averaged points (src/cuda.cu:387-446,736)
    from oracle.monitor import monitor
    expected = monitor(m, *d)
    assert abs(mon - expected) <= 1e-12 * abs(expected), (mon, expected)


def test_resident_restart_and_snapshot(gpu):
    # tests/test_research.cpp:740-761
    lp = tiny(2, 1, [(0, 0, 1.0), (0, 1, 1.0)])
    lp.lb[:] = 0
    lp.ub[:] = 5
    lp.rl = np.array([3.0])
    lp.c = np.array([1.0, 2.0])
    r = gpu.PdhgBackend(lp)
    r.advance(20, .1, .1)
    rx, ry, ra, rb = r.candidates()
    state = r.snapshot()
    assert r.reset_candidate(True)
    r.advance(20, .1, .1)
    sx, sy, _, _ = r.candidates()
    r.restore(state)
    r.reset(ra, rb)
    r.advance(20, .1, .1)
    rx, ry, _, _ = r.candidates()
    near(rx, sx, 1e-12)
    near(ry, sy, 1e-12)


@pytest.mark.parametrize("name,tol", [("steps_lp_adaptive", 1e-10), ("steps_lp_fixed", 1e-10),
                                      ("steps_qp", 1e-10), ("steps_skewed", 1e-9)])
@pytest.mark.parametrize("graphs", [False, True])
def test_golden_step_parity(gpu, name, tol, graphs):
    """Engine vs the reference's own CPU trajectory (golden fixtures)."""
    model, d = load_golden(name)
    kw = json.loads(str(d["options"]))
    kw.pop("restarts", None)
    g = gpu.PdhgBackend(model, graphs=graphs, **kw)
    done = 0
    for k in range(len(d["progress"])):
        done = advance_to(g, done + int(d["progress"][k]), float(d["tau"]), float(d["sigma"]),
                          done)
        assert g.rejected_steps() == d["rejected"][k]
        x, y, xa, ya = g.candidates()
        near(x, d["x"][k], tol)
        near(y, d["y"][k], tol)
        near(xa, d["xa"][k], tol)
        near(ya, d["ya"][k], tol)


def test_golden_halpern_restart_request(gpu):
    model, d = load_golden("steps_lp_halpern")
    g = gpu.PdhgBackend(model, halpern=True, reflection=0.5, residual_restarts=True)
    for k in range(2):
        assert g.advance(5, float(d["tau"]), float(d["sigma"])) == d["progress"][k]
        x, y, xa, ya = g.candidates()
        near(x, d["x"][k], 1e-10)
        near(y, d["y"][k], 1e-10)
    # The tenth accepted step raises the restart request (the CPU then returns one
    # step per call, progress [5, 5, 1, ...]).  Like the reference CUDA backend
    # (src/cuda.cu:298-301), the device freezes every further trial until the
    # driver restarts.
    assert list(d["progress"][:3]) == [5, 5, 1]
    assert g.restart_requested()
    x0, y0, _, _ = g.candidates()
    assert g.advance(5, float(d["tau"]), float(d["sigma"])) == 0
    x1, y1, _, _ = g.candidates()
    assert np.array_equal(x0, x1) and np.array_equal(y0, y1)
    g.reset_candidate(True)
    assert not g.restart_requested()
    assert g.advance(5, float(d["tau"]), float(d["sigma"])) == 5


def test_sparse_qp_parity(gpu, oracle):
    m = sparse_qp_model()
    cpu = oracle.model(m).backend(np.zeros(2), np.zeros(1))
    g = gpu.PdhgBackend(m)
    for _ in range(10):
        assert cpu.advance(7, 0.3, 0.3) == g.advance(7, 0.3, 0.3)
        for u, w in zip(g.candidates(), cpu.candidates()):
            near(u, w)


@pytest.mark.parametrize("seed", [1, 2])
def test_random_lp_adaptive_parity(gpu, oracle, seed):
    """Adaptive steps on a power-law LP with rows of up to 6,000 entries and row
    scales over four decades.  Tolerance 1e-8 relative after 40 accepted steps:
    the device adds a long row's segments and the step rule's sums in a fixed
    tree, the CPU loop adds them one by one, and the adaptive step factor (a
    ratio of those sums) carries those last-bit differences from one step to
    the next."""
    m = synth.power_law_lp(m=4000, n=8000, nnz=80000, seed=seed, len_hi=6000)
    cpu = oracle.model(m).backend(np.zeros(m.n), np.zeros(m.m), adaptive=True)
    g = gpu.PdhgBackend(m, adaptive=True, graphs=True)
    done = 0
    for _ in range(4):
        done = advance_to(g, done + cpu.advance(10, 0.01, 0.01), 0.01, 0.01, done)
        assert g.rejected_steps() == cpu.rejected_steps()
        for u, w in zip(g.candidates(), cpu.candidates()):
            near(u, w, 1e-8)


def test_fp32_precision_tracks_fp64(gpu):
    """FP32 matrix values, FP32 gathers and accumulation; iterates stay FP64.
    Tolerance: 1e-4 relative to the FP64 engine after 40 fixed steps."""
    m = synth.random_lp(m=500, n=1200, per_col=4, seed=8)
    a = gpu.PdhgBackend(m, precision="fp64")
    b = gpu.PdhgBackend(m, precision="fp32")
    a.advance(40, 0.05, 0.05)
    b.advance(40, 0.05, 0.05)
    for u, w in zip(b.candidates(), a.candidates()):
        near(u, w, 1e-4)


def test_empty_and_degenerate_shapes(gpu, oracle):
    # no rows; a row without entries; an all-zero column
    m = tiny(3, 2, [(0, 0, 1.0), (0, 2, -2.0)])
    m.c = np.array([1.0, -1.0, 0.5])
    m.rl = np.array([-1.0, -math.inf])
    m.ru = np.array([2.0, math.inf])
    cpu = oracle.model(m).backend(np.zeros(3), np.zeros(2), adaptive=True)
    g = gpu.PdhgBackend(m, adaptive=True)
    done = 0
    for _ in range(5):
        done = advance_to(g, done + cpu.advance(3, 0.2, 0.2), 0.2, 0.2, done)
        assert g.rejected_steps() == cpu.rejected_steps()
        for u, w in zip(g.candidates(), cpu.candidates()):
            near(u, w)
    e = tiny(4, 0, [])
    e.c = np.array([1.0, -1.0, 0.0, 2.0])
    cpu = oracle.model(e).backend(np.zeros(4), np.zeros(0))
    g = gpu.PdhgBackend(e)
    assert cpu.advance(5, 0.5, 0.5) == g.advance(5, 0.5, 0.5)
    near(g.candidates()[0], cpu.candidates()[0])


def test_fixed_step_nonfinite_is_an_error(gpu):
    m = tiny(1, 1, [(0, 0, 1e300)])
    m.lb[:] = -math.inf
    m.ub[:] = math.inf
    m.c[:] = 1e300
    m.rl[:] = m.ru[:] = 1
    g = gpu.PdhgBackend(m)
    with pytest.raises(gpu.EngineError) as e:
        for _ in range(5):
            g.advance(10, 1e10, 1e10)
    assert "stalled or produced nonfinite" in str(e.value)


def test_very_long_rows_and_columns_parity(gpu, oracle):
    """A row of 20000 entries (split across chunks, combined through slots) and a
    dense column (a long row of A^T), against the oracle."""
    rng = np.random.default_rng(17)
    n, m = 20000, 300
    rows = [np.zeros(n, dtype=np.int64)]          # row 0: every column
    cols = [np.arange(n, dtype=np.int64)]
    for i in range(1, m):
        k = rng.integers(2, 12)
        rows.append(np.full(k, i, dtype=np.int64))
        cols.append(np.sort(rng.choice(n, k, replace=False)))
    r = np.concatenate(rows)
    c = np.concatenate(cols)
    dense_col = 7                                   # column 7 in every row
    extra = np.arange(1, m)
    keep = ~np.isin(extra, r[c == dense_col])
    r = np.concatenate([r, extra[keep]])
    c = np.concatenate([c, np.full(keep.sum(), dense_col)])
    v = rng.standard_normal(r.size)
    order = np.lexsort((c, r))
    r, c, v = r[order], c[order], v[order]
    ptr = np.zeros(m + 1, dtype=np.int64)
    np.cumsum(np.bincount(r, minlength=m), out=ptr[1:])
    x0 = rng.uniform(0, 1, n)
    model = synth.Model(m=m, n=n, ptr=ptr, idx=c, val=v, c=rng.standard_normal(n), q=np.zeros(n),
                        lb=np.zeros(n), ub=np.ones(n), rl=np.full(m, -np.inf), ru=np.zeros(m))
    model.ru = synth.csr_matvec(ptr, c, v, x0, m) + 0.5
    cpu = oracle.model(model).backend(np.zeros(n), np.zeros(m), adaptive=True)
    for graphs in (False, True):
        g = gpu.PdhgBackend(model, adaptive=True, graphs=graphs)
        done = 0
        c2 = oracle.model(model).backend(np.zeros(n), np.zeros(m), adaptive=True)
        for _ in range(3):
            done = advance_to(g, done + c2.advance(5, 0.001, 0.001), 0.001, 0.001, done)
            assert g.rejected_steps() == c2.rejected_steps()
            for u, w in zip(g.candidates(), c2.candidates()):
                near(u, w, 1e-9)


@pytest.mark.parametrize("seed", [1, 2])
def test_compact_csr_matches_host_compaction(gpu, seed):
    """cuda_compact_matrix on the GPU against the host restriction of the same
    CSR: kept rows in order, kept columns renumbered, entries in source order --
    bit-identical (an integer / byte operation).  Includes empty rows, rows of
    more than 32 entries and a dropped-everything row."""
    rng = np.random.default_rng(seed)
    m = synth.power_law_lp(m=3000, n=6000, nnz=60000, seed=seed, len_hi=2000)
    kept = np.sort(rng.choice(m.m, 2000, replace=False))
    keep_col = rng.random(m.n) < 0.7
    cmap = np.where(keep_col, np.cumsum(keep_col) - 1, -1)
    out_cols = int(keep_col.sum())
    ptr, idx, val = gpu.compact_csr(m.ptr, m.idx, m.val, m.n, kept, cmap, out_cols)
    want_ptr, want_idx, want_val = [0], [], []
    for i in kept:
        cols = m.idx[m.ptr[i]:m.ptr[i + 1]]
        vals = m.val[m.ptr[i]:m.ptr[i + 1]]
        sel = cmap[cols] >= 0
        want_idx.extend(cmap[cols[sel]].tolist())
        want_val.extend(vals[sel].tolist())
        want_ptr.append(len(want_idx))
    assert np.array_equal(ptr, want_ptr)
    assert np.array_equal(idx, want_idx)
    assert np.array_equal(val.view(np.int64), np.array(want_val).view(np.int64))


def test_compact_csr_rejects_bad_maps(gpu):
    m = synth.random_lp(m=50, n=80, per_col=3, seed=1)
    cmap = np.arange(m.n)
    with pytest.raises(gpu.EngineError, match="row map"):
        gpu.compact_csr(m.ptr, m.idx, m.val, m.n, [3, 2], cmap, m.n)
    bad = cmap.copy()
    bad[5] = 2  # not increasing
    with pytest.raises(gpu.EngineError, match="column map"):
        gpu.compact_csr(m.ptr, m.idx, m.val, m.n, [0, 1], bad, m.n)


def _propagation_case(seed):
    """A random sparse model with mixed-sign rows, equality and one-sided rows,
    free and boxed columns, and a random half of the columns integer."""
    rng = np.random.default_rng(seed)
    m = synth.random_lp(m=400, n=900, per_col=4, seed=seed)
    lb, ub = m.lb.copy(), m.ub.copy()
    free = rng.random(m.n) < 0.1
    lb[free], ub[free] = -np.inf, np.inf
    m.rl = np.where(rng.random(m.m) < 0.5, m.rl - 0.5, -np.inf)
    m.ru = m.ru + rng.uniform(0, 2, m.m)
    integer = (rng.random(m.n) < 0.5).astype(np.int32)
    return m, integer, lb, ub


@pytest.mark.parametrize("seed", [3, 4, 5])
@pytest.mark.parametrize("passes", [1, 5])
def test_propagate_bounds_matches_oracle(gpu, oracle, seed, passes):
    """cuda_propagate_integer_bounds on the GPU against the oracle's sequential
    restatement with the rounding mode switched per operation: bounds and the
    feasibility verdict bit-identical (each row's sums keep their order; the
    tightest proposal per column wins whatever the arrival order)."""
    m, integer, lb, ub = _propagation_case(seed)
    ok_g, lb_g, ub_g = gpu.propagate_bounds(m, integer, lb, ub, passes)
    ok_o, lb_o, ub_o = oracle.propagate_bounds(m, integer, lb, ub, passes)
    assert ok_g == ok_o
    assert np.array_equal(lb_g.view(np.int64), lb_o.view(np.int64))
    assert np.array_equal(ub_g.view(np.int64), ub_o.view(np.int64))
    assert np.sum(lb_g > lb) + np.sum(ub_g < ub) > 0  # something was tightened


def test_propagate_bounds_detects_infeasible_row(gpu, oracle):
    m, integer, lb, ub = _propagation_case(6)
    m.rl = m.rl.copy()
    m.rl[7] = 1e9  # no point in the box reaches it
    ok_g = gpu.propagate_bounds(m, integer, lb, ub, 3)[0]
    assert ok_g is False and oracle.propagate_bounds(m, integer, lb, ub, 3)[0] is False


def _newton_system(n, seed=11):
    """A nonsymmetric, diagonally dominant sparse system (CSR and dense)."""
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), 6)
    cols = rng.integers(0, n, rows.size)
    vals = rng.standard_normal(rows.size)
    dense = np.zeros((n, n))
    np.add.at(dense, (rows, cols), vals)
    dense[np.arange(n), np.arange(n)] += 8 + np.abs(dense).sum(1)
    nz = dense != 0
    ptr = np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int64)
    idx = np.nonzero(nz)[1].astype(np.int64)
    return ptr, idx, dense[nz], dense, rng.standard_normal(n)


@pytest.mark.parametrize("fp32", [False, True])
def test_linear_solve_bicgstab(gpu, fp32):
    """cuda_linear_solve's BiCGSTAB on a nonsymmetric, diagonally dominant sparse
    system: converged, and the solution within the target the reference sets
    (1e-10 relative residual in FP64, 1e-6 with FP32 values) of the dense solve."""
    ptr, idx, val, dense, rhs = _newton_system(3000)
    x, ok = gpu.linear_solve(ptr, idx, val, rhs, fp32_matrix=fp32)
    assert ok
    want = np.linalg.solve(dense, rhs)
    tol = 1e-5 if fp32 else 1e-9
    assert np.max(np.abs(x - want)) <= tol * (1 + np.max(np.abs(want)))
    if not fp32:
        assert np.linalg.norm(dense @ x - rhs) <= 1e-10 * (1 + np.linalg.norm(rhs)) * 10


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
def test_panel_path_multi_panel_parity(gpu, oracle, precision):
    """A's long rows by column panel (the dual SpMV's panel kernel) with more
    than one panel: 100,000 columns are several panels of the FP64 dx slice a
    CTA holds (two of the FP32 one).  Fixed steps against the oracle, 1e-10
    relative in FP64 over 60 trials: a long row is summed per panel in CSR
    order and the panel sums are added in panel order, where the CPU adds the
    whole row in CSR order.  With FP32 matrices the oracle gets the same
    FP32-rounded values (MIXED: FP64 gathers and sums, 1e-10) or the FP32
    engine is held to 1e-4 (FP32 gathers and sums)."""
    m = synth.power_law_lp(m=20000, n=100000, nnz=500000, seed=3, len_hi=5000)
    if precision != "fp64":
        m.val = m.val.astype(np.float32).astype(np.float64)
    g = gpu.PdhgBackend(m, graphs=True, precision=precision)
    info = g.layout_info()
    assert info["panels"] >= 2 and info["panel_rows"] > 0, info
    assert info["kernels_per_trial"] == 3
    cpu = oracle.model(m).backend(np.zeros(m.n), np.zeros(m.m))
    tol = 1e-4 if precision == "fp32" else 1e-10
    tau, sigma = step_sizes(m)
    for _ in range(3):
        assert cpu.advance(20, tau, sigma) == g.advance(20, tau, sigma)
        for u, w in zip(g.candidates(), cpu.candidates()):
            near(u, w, tol)


def test_panel_path_single_panel_runs(gpu, oracle):
    """With every column in one panel a long row's partials are its runs: its
    entries in CSR order, cut into pieces of 64 or more where one lane would
    otherwise carry far more than its share, each summed sequentially and then
    added in CSR order.  Rows of up to 3,000 entries on a 3,000-row LP are cut
    (more runs than long rows); fixed-step trajectories agree with the CPU's
    sequential row sums to 1e-12 over 50 trials."""
    m = synth.power_law_lp(m=3000, n=6000, nnz=60000, seed=4, len_hi=3000)
    g = gpu.PdhgBackend(m, graphs=True)
    info = g.layout_info()
    assert info["panels"] == 1 and info["panel_rows"] > 0, info
    assert info["panel_runs"] > info["panel_rows"], info
    cpu = oracle.model(m).backend(np.zeros(m.n), np.zeros(m.m))
    tau, sigma = step_sizes(m)
    assert cpu.advance(50, tau, sigma) == g.advance(50, tau, sigma)
    for u, w in zip(g.candidates(), cpu.candidates()):
        near(u, w, 1e-12)


def test_trajectory_parity_above_openmp_threshold(gpu, reference):
    """Step by step against the reference's own CpuBackend (oracle/_ref, all host
    threads) above its OpenMP threshold (10,000 rows or columns,
    src/cpu.cpp:105,123,134), where its step-rule sums are split over threads:
    a power-law LP of 50,000 x 100,000 with 1,000,000 nonzeros and rows of up to
    5,000 entries (several column panels on the device).  Adaptive steps,
    compared at equal accepted counts; tolerance 1e-8 relative after 40
    accepted steps, as for the oracle runs on smaller power-law LPs: both sides
    group the sums differently and the adaptive step factor carries the
    last-bit differences forward."""
    import os
    os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count() or 1))
    m = synth.power_law_lp(m=50000, n=100000, nnz=1_000_000, seed=6, len_hi=5000)
    assert int(np.diff(m.ptr).max()) > 4000
    cpu = reference.model(m).backend(np.zeros(m.n), np.zeros(m.m), adaptive=True)
    g = gpu.PdhgBackend(m, adaptive=True, graphs=True)
    assert g.layout_info()["panels"] >= 2
    tau, sigma = step_sizes(m)
    done = 0
    for _ in range(4):
        done = advance_to(g, done + cpu.advance(10, tau, sigma), tau, sigma, done)
        assert g.rejected_steps() == cpu.rejected_steps()
        for u, w in zip(g.candidates(), cpu.candidates()):
            near(u, w, 1e-8)


@pytest.mark.parametrize("graphs", [False, True])
def test_profiled_trials_are_ordinary_trials(gpu, graphs):
    """nk_pdhg_profile_kernels times the kernels of real trials (with graphs on,
    replays of one captured trial whose events are graph nodes): its trials
    advance the iterate bit for bit as advance() does, and every kernel time is
    positive, the panel kernel's too on an LP with panels."""
    m = synth.power_law_lp(m=20000, n=100000, nnz=500000, seed=3, len_hi=5000)
    tau, sigma = step_sizes(m)
    a = gpu.PdhgBackend(m, adaptive=True, graphs=graphs)
    b = gpu.PdhgBackend(m, adaptive=True, graphs=graphs)
    assert a.layout_info()["panels"] >= 2
    primal, panel, dual = a.profile_kernels(30, tau, sigma)
    assert primal > 0 and panel > 0 and dual > 0
    b.advance(30, tau, sigma)
    for u, w in zip(a.candidates(), b.candidates()):
        assert np.array_equal(u, w)


def resident_model(kind):
    if kind == "one row":
        m = tiny(3, 1, [(0, 0, 1.0), (0, 1, -2.0), (0, 2, 0.5)])
        m.c[:] = [1.0, -1.0, 0.5]
        m.rl[:] = m.ru[:] = 3
        return m
    if kind == "empty rows and columns":
        m = synth.random_lp(m=70, n=131, per_col=2, seed=5)
        keep = (m.idx % 7 != 0) & (np.repeat(np.arange(m.m), np.diff(m.ptr)) % 5 != 0)
        counts = np.add.reduceat(np.r_[keep, 0].astype(np.int64), m.ptr[:-1]) * (np.diff(m.ptr) > 0)
        m.ptr = np.concatenate([[0], np.cumsum(counts)])
        m.idx, m.val = m.idx[keep], m.val[keep]
        return m
    if kind == "dense column":  # 400 entries: a split row of A^T
        rows, cols = 400, 97
        rng = np.random.default_rng(6)
        entries = sorted({(i, 3) for i in range(rows)} |
                         {(i, int(j)) for i in range(rows) for j in rng.integers(0, cols, 3)})
        m = tiny(cols, rows, [(i, j, float(rng.standard_normal())) for i, j in entries])
        m.c[:] = rng.standard_normal(cols)
        m.rl[:] = m.ru[:] = rng.standard_normal(rows)
        return m
    shapes = {"chunk": (32, 64), "chunk and one": (33, 65), "small": (2000, 5000),
              "unstaged entries": (60000, 130001), "unstaged": (100003, 200001)}
    m, n = shapes[kind]
    return synth.random_lp(m=m, n=n, per_col=5, seed=7)


@pytest.mark.parametrize("method", ["adaptive", "rejecting", "fixed", "halpern", "quadratic",
                                    "mixed"])
@pytest.mark.parametrize("kind", ["one row", "empty rows and columns", "dense column", "chunk",
                                  "chunk and one", "small", "unstaged entries", "unstaged"])
def test_resident_trials_match_the_kernel_path(gpu, kind, method):
    """advance() of a small or medium model runs its trials in one launch; the
    profiled trials run as kernels of their own.  Both add every sum in the same
    order, so the points agree bit for bit, over several calls, with rejected
    trials, Halpern commits, a diagonal quadratic term and FP32 values."""
    m = resident_model(kind)
    if method == "quadratic":
        m.q = np.random.default_rng(8).uniform(0.1, 1.0, m.n)
    tau, sigma = step_sizes(m)
    if method == "rejecting":
        tau, sigma = 40 * tau, 40 * sigma
    options = dict(adaptive=method not in ("fixed", "halpern"), graphs=True,
                   precision="mixed" if method == "mixed" else "fp64")
    if method == "halpern":
        options.update(halpern=True, reflection=0.5, residual_restarts=True)
    a, b = gpu.PdhgBackend(m, **options), gpu.PdhgBackend(m, **options)
    for count in (1, 2, 30):
        a.advance(count, tau, sigma)
        b.profile_kernels(count, tau, sigma)
        for u, w in zip(a.candidates(), b.candidates()):
            assert np.array_equal(u, w)
    assert a.rejected_steps() == b.rejected_steps()
    if method == "rejecting" and kind == "small":
        assert a.rejected_steps() > 0


def test_adaptive_steps_keep_the_panels_order(gpu):
    """Adaptive steps amplify rounding, so a model with column panels runs them
    under advance() too: its points are the profiled panel kernels', bit for bit."""
    m = synth.power_law_lp(m=3000, n=6000, nnz=60000, seed=4, len_hi=3000)
    tau, sigma = step_sizes(m)
    a, b = (gpu.PdhgBackend(m, adaptive=True, graphs=True) for _ in range(2))
    assert a.layout_info()["panels"] > 0
    a.advance(80, tau, sigma)
    b.profile_kernels(80, tau, sigma)
    for u, w in zip(a.candidates(), b.candidates()):
        assert np.array_equal(u, w)


def test_panel_engines_of_different_widths_coexist(gpu):
    """Two engines whose panels differ in width: the kernel's shared-memory limit
    belongs to both, so the wider one still runs after the narrower was built."""
    wide = synth.power_law_lp(m=20000, n=100000, nnz=500000, seed=3, len_hi=5000)
    narrow = synth.power_law_lp(m=3000, n=6000, nnz=60000, seed=4, len_hi=3000)
    a = gpu.PdhgBackend(wide)
    b = gpu.PdhgBackend(narrow)
    assert a.layout_info()["panel_width"] > b.layout_info()["panel_width"] > 0
    for g, m in ((a, wide), (b, narrow)):
        tau, sigma = step_sizes(m)
        assert g.advance(5, tau, sigma) == 5


def sparse_q(n, kind):
    """Symmetric CSR of a positive semidefinite Q: a few rows of a rank-four term,
    a tridiagonal matrix, or one dense row and column."""
    rng = np.random.default_rng(9)
    if kind == "low rank":
        return synth.sparse_qp_terms(rng, n)[:3]
    dense = np.zeros((n, n))
    k = np.arange(n)
    if kind == "tridiagonal":
        dense[k, k] = 2.0
        dense[k[1:], k[:-1]] = dense[k[:-1], k[1:]] = -1.0
    else:
        dense[5, :] = dense[:, 5] = 0.01
        dense[k, k] = 1.0
    ptr = np.r_[0, np.cumsum(np.count_nonzero(dense, axis=1))].astype(np.int64)
    r, c = np.nonzero(dense)
    return ptr, c.astype(np.int64), dense[r, c]


@pytest.mark.parametrize("halpern", [False, True])
@pytest.mark.parametrize("kind", ["low rank", "tridiagonal", "dense row"])
def test_sparse_q_rows_shared_by_lanes(gpu, oracle, kind, halpern):
    """Q x by groups of lanes: the resident trials and the kernel path agree bit for
    bit, and both with the oracle's sequential row sums to 1e-11 (a row of up to
    600 terms of one size rounds within 600 ulp, 1.4e-13, per trial)."""
    m = synth.random_lp(m=300, n=600, per_col=4, seed=10)
    m.qptr, m.qidx, m.qval = sparse_q(m.n, kind)
    tau, sigma = step_sizes(m)
    options = dict(halpern=halpern, reflection=0.5 if halpern else 0.0)
    a, b = gpu.PdhgBackend(m, graphs=True, **options), gpu.PdhgBackend(m, graphs=True, **options)
    cpu = oracle.model(m).backend(np.zeros(m.n), np.zeros(m.m), **options)
    # the step sizes a QP's advance would reduce its own to are the caller's here
    scale = 0.01
    for count in (1, 30):
        a.advance(count, scale * tau, scale * sigma)
        b.profile_kernels(count, scale * tau, scale * sigma)
        cpu.advance(count, scale * tau, scale * sigma)
        for u, w, z in zip(a.candidates(), b.candidates(), cpu.candidates()):
            assert np.array_equal(u, w)
            near(u, z)


@pytest.mark.parametrize("n", [1, 31, 257, 40_000, 160_001])
@pytest.mark.parametrize("wide", [False, True])
def test_linear_solve_sizes(gpu, n, wide):
    """BiCGSTAB in one kernel: rows of 1 to 6 entries (8 lanes a row) and with one
    row of 50 (32 lanes, more than one stride), sizes below and above what the
    grid's threads hold one element each of.  K = 4 I + E with at most 0.5 in
    absolute sums off the diagonal per row, so ||K^-1|| <= 1/3.5 in the maximum
    norm: the answer is within (1e-10 (1 + |rhs|)) / 3.5 of the exact one."""
    rng = np.random.default_rng(n)
    rows = [np.repeat(np.arange(n), 5)]
    cols = [rng.integers(0, n, 5 * n)]
    if wide and n > 200:
        rows.append(np.full(50, n // 2))
        cols.append(rng.choice(n, 50, replace=False))
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    key = np.unique((rows * n + cols)[rows != cols])
    r, c = key // n, key % n
    off = rng.uniform(-1, 1, r.size) * 0.5 / np.maximum(1, np.bincount(r, minlength=n))[r]
    order = np.lexsort((np.r_[c, np.arange(n)], np.r_[r, np.arange(n)]))
    idx = np.r_[c, np.arange(n)][order].astype(np.int64)
    val = np.r_[off, np.full(n, 4.0)][order]
    ptr = np.r_[0, np.cumsum(np.bincount(r, minlength=n) + 1)].astype(np.int64)
    rhs = rng.standard_normal(n)
    for precondition in (True, False):
        x, ok = gpu.linear_solve(ptr, idx, val, rhs, precondition=precondition)
        assert ok
        residual = rhs - np.add.reduceat(val * x[idx], ptr[:-1])
        # the recurrence's residual met the target; its drift is rounding of a few dozen steps
        target = 1e-10 * (1 + np.linalg.norm(rhs))
        assert np.linalg.norm(residual) <= 2 * target
    with pytest.raises(TimeoutError):
        gpu.linear_solve(ptr, idx, val, rhs, time_limit=0.0)


@pytest.mark.parametrize("rows,per", [(1, 3), (33, 1), (64, 20), (65, 21), (200, 60), (500, 9)])
def test_propagate_bounds_row_groups(gpu, oracle, rows, per):
    """Bound propagation by groups of 32 rows: a last group of one row, empty rows,
    zero coefficients, infinite bounds, groups of exactly the 640 entries that fit
    a warp's buffers and of more, which a lane walks; bit-identical to the
    sequential restatement."""
    rng = np.random.default_rng(100 * rows + per)
    n = 3 * rows + per
    entries = [(i, int(j), float(v)) for i in range(rows) if rows == 64 or i % 11 != 5
               for j, v in zip(np.sort(rng.choice(n, per, replace=False)),
                               np.round(rng.standard_normal(per), 1))]
    m = tiny(n, rows, entries)
    lb, ub = rng.uniform(-5, 0, n), rng.uniform(0, 40, n)
    lb[::13], ub[::17] = -np.inf, np.inf
    m.rl, m.ru = rng.uniform(-30, -10, rows), rng.uniform(10, 30, rows)
    m.rl[::5] = -np.inf
    integer = (np.arange(n) % 3 == 0).astype(np.int32)
    got = gpu.propagate_bounds(m, integer, lb, ub, 4)
    want = oracle.propagate_bounds(m, integer, lb, ub, 4)
    assert got[0] == want[0]
    for u, w in zip(got[1:], want[1:]):
        assert np.array_equal(u.view(np.int64), w.view(np.int64))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nnz,len_hi,panels", [(1_600_000, 5000, False), (1_600_000, 9000, False),
                                               (9_000_000, 9000, True)])
def test_long_rows_past_the_resident_size(gpu, oracle, nnz, len_hi, panels, precision):
    """Models too large for the resident trials: long rows as split rows where they
    hold fewer than 4 M entries (rows of more than 8,192 across chunks), by column
    panel above; against the CPU's sequential sums over 20 fixed-step trials.  A row
    of 9,000 terms regrouped rounds within 9,000 ulp of its terms' magnitude,
    2e-12, per trial: 1e-10 in all."""
    m = synth.power_law_lp(m=60_000, n=40_000, nnz=nnz, seed=11, len_lo=2 if not panels else 100,
                           len_hi=len_hi)
    if precision == "mixed":
        m.val = m.val.astype(np.float32).astype(np.float64)
    g = gpu.PdhgBackend(m, graphs=True, precision=precision)
    assert (g.layout_info()["panels"] > 0) == panels
    cpu = oracle.model(m).backend(np.zeros(m.n), np.zeros(m.m))
    tau, sigma = step_sizes(m)
    assert cpu.advance(20, tau, sigma) == g.advance(20, tau, sigma)
    for u, w in zip(g.candidates(), cpu.candidates()):
        near(u, w, 1e-10)


def test_resident_trials_from_several_threads(gpu):
    """Four engines advanced from four threads at once, each on its own stream: the
    resident grids take every SM, so they must run one after the other, whole; each
    engine ends where it ends alone, bit for bit."""
    import threading
    models = [synth.random_lp(m=m, n=n, per_col=4, seed=m) for m, n in
              ((400, 1000), (9000, 20000), (2000, 5000), (20000, 50001))]
    steps = [step_sizes(m) for m in models]

    def run(k, out):
        g = gpu.PdhgBackend(models[k], adaptive=True, graphs=True)
        for _ in range(25):
            g.advance(40, *steps[k])
        out[k] = g.candidates()

    alone, together = {}, {}
    for k in range(4):
        run(k, alone)
    threads = [threading.Thread(target=run, args=(k, together)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(together) == 4
    for k in range(4):
        for u, w in zip(alone[k], together[k]):
            assert np.array_equal(u, w)


def test_resident_trials_frozen_in_mid_chunk(gpu):
    """A Halpern restart requested by the tenth of 40 trials freezes the other 30, and
    the next launches' barriers start from zero again: bit for bit the trials that
    run as kernels of their own, over several restarts and chunk lengths."""
    model, d = load_golden("steps_lp_halpern")
    tau, sigma = float(d["tau"]), float(d["sigma"])
    options = dict(halpern=True, reflection=0.5, residual_restarts=True, graphs=True)
    a, b = gpu.PdhgBackend(model, **options), gpu.PdhgBackend(model, **options)
    requests = 0
    for count in (40, 40, 1, 2, 3, 40, 17, 40):
        a.advance(count, tau, sigma)
        b.profile_kernels(count, tau, sigma)
        for u, w in zip(a.candidates(), b.candidates()):
            assert np.array_equal(u, w)
        if a.restart_requested():
            requests += 1
            for g in (a, b):
                g.reset_candidate(True)
    assert requests >= 1


@pytest.mark.parametrize("method", ["adaptive", "halpern", "mixed"])
@pytest.mark.parametrize("split", [False, True])
def test_resident_trials_with_unstaged_bounds(gpu, split, method):
    """The largest resident models keep only the iterate in shared memory and read
    bounds and costs where they lie: a last chunk of one column (31 lanes past the
    end of c), without and with columns long enough to be split (400 entries; the
    other columns then start at a chunk of their own).  Bit for bit the trials that
    run as kernels of their own."""
    m = synth.random_lp(m=100_003, n=270_017 + (2 if split else 0), per_col=5, seed=12)
    if split:
        rng = np.random.default_rng(13)
        rows = np.repeat(np.arange(m.m), np.diff(m.ptr))
        extra = [rng.choice(m.m, 400, replace=False) * m.n + j for j in (7, 200_000)]
        key, first = np.unique(np.concatenate([rows * m.n + m.idx, *extra]), return_index=True)
        m.val = np.concatenate([m.val, rng.standard_normal(800)])[first]
        m.idx = key % m.n
        m.ptr = np.r_[0, np.cumsum(np.bincount(key // m.n, minlength=m.m))].astype(np.int64)
    tau, sigma = step_sizes(m)
    options = dict(adaptive=method != "halpern", halpern=method == "halpern", graphs=True,
                   precision="mixed" if method == "mixed" else "fp64")
    a, b = gpu.PdhgBackend(m, **options), gpu.PdhgBackend(m, **options)
    info = a.layout_info()
    assert info["resident"] and info["resident_stage"] == 0, info
    for count in (1, 2, 30):
        a.advance(count, tau, sigma)
        b.profile_kernels(count, tau, sigma)
        for u, w in zip(a.candidates(), b.candidates()):
            assert np.array_equal(u, w)


def test_a_wait_given_up_is_reported_once(gpu):
    """After a trial launch that gave up a wait (marked here as one leaves it),
    advance() of several queued launches and profile_kernels() report it without
    having run a trial, and the calls after that run from whole counters: bit for bit
    an engine that never failed."""
    m = synth.power_law_lp(m=3000, n=6000, nnz=60000, seed=4, len_hi=3000)
    tau, sigma = step_sizes(m)
    a, b = gpu.PdhgBackend(m, graphs=True), gpu.PdhgBackend(m, graphs=True)
    info = a.layout_info()
    assert info["resident"] and info["panels"] > 0, info
    for call in (lambda: a.advance(9000, tau, sigma), lambda: a.profile_kernels(5, tau, sigma)):
        a.advance(7, tau, sigma)
        b.advance(7, tau, sigma)
        gpu.check(gpu.library().nk_pdhg_mark_fault(a._h))
        with pytest.raises(gpu.EngineError) as e:
            call()
        assert e.value.status == "CUDA"
        assert a.advance(7, tau, sigma) == b.advance(7, tau, sigma) == 7
        for u, w in zip(a.candidates(), b.candidates()):
            assert np.array_equal(u, w)
    wide = gpu.PdhgBackend(m, indices="64")
    with pytest.raises(gpu.EngineError):
        gpu.check(gpu.library().nk_pdhg_mark_fault(wide._h))


def test_slot_limits_of_large_engines_coexist(gpu):
    """The step rule's slots of 20 M rows take 66 KB of shared memory a CTA, those of
    15 M rows 50 KB: the kernel's limit belongs to both engines, so the larger one
    still runs after the smaller was built."""
    def model(m, n):
        val = np.where(np.arange(m) % 2 == 0, 1.0, -1.0)
        ptr, idx = np.arange(m + 1, dtype=np.int64), np.arange(m, dtype=np.int64) % n
        return synth.Model(m=m, n=n, ptr=ptr, idx=idx, val=val, c=np.ones(n), q=np.zeros(n),
                           lb=np.zeros(n), ub=np.ones(n), rl=np.zeros(m), ru=np.ones(m),
                           name="rows of one entry", x0=np.zeros(n))
    large = gpu.PdhgBackend(model(20_000_000, 1_000_000))
    small = gpu.PdhgBackend(model(15_000_000, 1_000_000))
    assert large.advance(2, 0.01, 0.01) == 2
    assert small.advance(2, 0.01, 0.01) == 2


def test_kernels_of_a_trial_are_counted(gpu):
    """The launches of a trial that runs as kernels of its own: the primal and the
    dual one, Q x of a sparse Q with long rows, and Halpern's commit."""
    m = synth.random_lp(m=300, n=600, per_col=4, seed=10)
    m.qptr, m.qidx, m.qval = sparse_q(m.n, "low rank")
    assert m.qptr[-1] > 24 * np.count_nonzero(np.diff(m.qptr))
    assert gpu.PdhgBackend(m).layout_info()["kernels_per_trial"] == 3
    assert gpu.PdhgBackend(m, halpern=True).layout_info()["kernels_per_trial"] == 4
    assert gpu.PdhgBackend(sparse_qp_model()).layout_info()["kernels_per_trial"] == 2
    m = synth.random_lp(m=70, n=131, per_col=2, seed=5)
    assert gpu.PdhgBackend(m).layout_info()["kernels_per_trial"] == 2
    assert gpu.PdhgBackend(m, halpern=True).layout_info()["kernels_per_trial"] == 3


def panel_model(kind, precision="fp64"):
    """A model whose long rows lie in several column panels, or cut into runs in one."""
    m = (synth.power_law_lp(m=20000, n=100000, nnz=500000, seed=3, len_hi=5000)
         if kind == "several panels" else
         synth.power_law_lp(m=3000, n=6000, nnz=60000, seed=4, len_hi=3000))
    if precision == "mixed":
        m.val = m.val.astype(np.float32).astype(np.float64)
    return m


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["several panels", "cut runs"])
def test_panel_kernel_under_adaptive_steps(gpu, oracle, kind, precision):
    """The panel kernel against the oracle where advance() launches it: a small model's
    fixed steps run resident, without it, its adaptive steps never do.  A long row of
    up to 5,000 terms, regrouped, rounds within 5,000 ulp, 6e-13, a trial, and adaptive
    steps carry that forward about tenfold every eight trials: 1e-9 over 10 accepted
    steps, where a lost or doubled run moves the point by its share."""
    m = panel_model(kind, precision)
    g = gpu.PdhgBackend(m, adaptive=True, graphs=True, precision=precision)
    info = g.layout_info()
    assert not info["resident"] and info["kernels_per_trial"] == 3, info
    assert info["panels"] >= 2 if kind == "several panels" else \
        info["panels"] == 1 and info["panel_runs"] > info["panel_rows"], info
    cpu = oracle.model(m).backend(np.zeros(m.n), np.zeros(m.m), adaptive=True)
    tau, sigma = step_sizes(m)
    advance_to(g, cpu.advance(10, tau, sigma), tau, sigma)
    assert g.rejected_steps() == cpu.rejected_steps()
    for u, w in zip(g.candidates(), cpu.candidates()):
        near(u, w, 1e-9)


def test_adaptive_panel_engines_of_different_widths_coexist(gpu):
    """The panel kernel's shared-memory limit belongs to every engine: the one with wide
    panels still launches it after one with narrow panels was built."""
    models = [panel_model(kind) for kind in ("several panels", "cut runs")]
    wide, narrow = (gpu.PdhgBackend(m, adaptive=True) for m in models)
    info = [g.layout_info() for g in (wide, narrow)]
    assert info[0]["panel_width"] > info[1]["panel_width"] > 0
    assert not (info[0]["resident"] or info[1]["resident"])
    for g, m in zip((wide, narrow), models):
        assert g.advance(20, *step_sizes(m)) > 0


def long_row_system(kind):
    """Newton systems with rows of many entries, as (rows, cols, values, n): dense; 40
    full rows and columns at the end of short ones (two warps' rows); rows of 31 to
    65 and of 257 entries; and a saddle point whose zero block's rows hold 40 entries
    and no diagonal."""
    rng = np.random.default_rng(14)
    if kind == "saddle":
        m, per = 150, 40
        n = m * per
        h = rng.uniform(0.1, 10, n)
        # rows without a common column, of scales from 1e-3 to 1e3: the Schur
        # complement is diagonal, and with it exact BiCGSTAB needs a few steps
        a = rng.uniform(0.5, 2, n) * np.repeat(10.0 ** rng.uniform(-3, 3, m), per)
        i, j = n + np.repeat(np.arange(m), per), np.arange(n)
        return np.r_[j, i, j], np.r_[j, j, i], np.r_[h, a, a], n + m
    if kind == "dense":
        n = 300
        r, c = np.divmod(np.arange(n * n), n)
    elif kind == "arrow":
        n, full = 5000, 40
        r, c = np.repeat(np.arange(n), 3), rng.integers(0, n, 3 * n)
        i, j = np.repeat(np.arange(n - full, n), n), np.tile(np.arange(n), full)
        r, c = np.r_[r, i, j], np.r_[c, j, i]
    else:
        n = 2000
        lens = np.r_[np.arange(30, 65), 256, np.full(n - 36, 4)]
        r = np.repeat(np.arange(n), lens)
        c = np.concatenate([rng.choice(n, k, replace=False) for k in lens])
    key = np.unique((r * n + c)[r != c])
    r, c = key // n, key % n
    off = rng.uniform(-1, 1, r.size) * 0.5 / np.maximum(1, np.bincount(r, minlength=n))[r]
    return np.r_[r, np.arange(n)], np.r_[c, np.arange(n)], np.r_[off, np.full(n, 4.0)], n


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("kind", ["dense", "arrow", "edges", "saddle"])
def test_linear_solve_long_rows(gpu, kind, fp32):
    """Rows of more than 32 entries are products of a warp each, and their scales are
    summed by one in the rows' order.  Held to the stopping target, twice for the
    drift of the recurrence's residual over a few dozen steps; the saddle point's rows
    differ in scale by six orders, so it converges only with the right scales."""
    rows, cols, vals, n = long_row_system(kind)
    order = np.lexsort((cols, rows))
    ptr = np.r_[0, np.cumsum(np.bincount(rows, minlength=n))].astype(np.int64)
    idx, val = cols[order].astype(np.int64), vals[order]
    rhs = np.random.default_rng(15).standard_normal(n)
    x, ok = gpu.linear_solve(ptr, idx, val, rhs, fp32_matrix=fp32)
    assert ok
    if fp32:
        val = val.astype(np.float32).astype(np.float64)
    residual = rhs - np.add.reduceat(val * x[idx], ptr[:-1])
    assert np.linalg.norm(residual) <= 2 * (1e-6 if fp32 else 1e-10) * (1 + np.linalg.norm(rhs))
    if kind != "saddle":
        y, ok = gpu.linear_solve(ptr, idx, val, rhs, fp32_matrix=fp32, precondition=False)
        assert ok
        # two answers within the target, of a matrix with ||K^-1|| <= 1/3.5
        assert np.max(np.abs(x - y)) <= (1e-6 if fp32 else 1e-10) * (1 + np.linalg.norm(rhs))


def test_linear_solve_time_limit_within_a_launch(gpu):
    """The time limit is looked at before every iteration.  8 M unknowns on a periodic
    grid whose matrix is singular, so that no residual meets the target: 64 iterations
    take tens of milliseconds, one takes less than one, so a limit of 10 ms ends the
    call no more than 15 ms (several times the spread of its uploads) later than a
    limit of 0 does, the limit itself aside."""
    import time
    n = 8_000_000
    i = np.arange(n)
    idx = np.concatenate([(i + d) % n for d in (0, 1, -1, 200, -200, 40_000, -40_000)])
    idx = np.ascontiguousarray(idx.reshape(7, n).T).reshape(-1)
    val = np.tile([6.0, -1, -1, -1, -1, -1, -1], n)
    ptr = 7 * np.arange(n + 1, dtype=np.int64)
    rhs = np.random.default_rng(16).standard_normal(n)

    def seconds(limit):
        best = np.inf
        for _ in range(5):
            start = time.perf_counter()
            with pytest.raises(TimeoutError):
                gpu.linear_solve(ptr, idx, val, rhs, time_limit=limit)
            best = min(best, time.perf_counter() - start)
        return best

    assert seconds(0.01) - seconds(0.0) <= 0.01 + 0.015


def device_bytes_during(call):
    """call()'s result and the most device memory that was taken while it ran."""
    import threading
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    least, done = [before], threading.Event()

    def watch():
        while not done.wait(0.001):
            least[0] = min(least[0], torch.cuda.mem_get_info()[0])
    watcher = threading.Thread(target=watch)
    watcher.start()
    try:
        result = call()
    finally:
        done.set()
        watcher.join()
    return result, before - least[0]


def test_linear_solve_fp32_memory(gpu):
    """FP32 values take 4 bytes an entry on the device beside 8 for the index; the FP64
    ones they and the scales are formed from pass through 128 MB at a time.  40 M
    entries, three such parts, in rows of 41 and 601.  Columns differ in scale by six
    orders, so the solve converges only with every column's scale right."""
    n = 125_000
    rng = np.random.default_rng(17)
    lens = np.where(np.arange(n) % 2 == 0, 600, 40)
    row = np.repeat(np.arange(n), lens)
    col = (row + 1 + rng.integers(0, n - 1, row.size)) % n
    scale = (10.0 ** rng.uniform(-3, 3, n)).astype(np.float32).astype(np.float64)
    off = rng.uniform(-0.5, 0.5, row.size) / np.repeat(lens, lens)
    ptr = np.r_[0, np.cumsum(lens + 1)].astype(np.int64)
    idx = np.empty(ptr[-1], dtype=np.int64)
    val = np.empty(ptr[-1])
    first = np.zeros(ptr[-1], dtype=bool)
    first[ptr[:-1]] = True
    idx[first], idx[~first] = np.arange(n), col
    val[first], val[~first] = 4 * scale, off * scale[col]
    rhs = rng.standard_normal(n)
    gpu.linear_solve(ptr[:2], np.zeros(601, dtype=np.int64), np.ones(601), rhs[:1],
                     fp32_matrix=True)  # context and kernels
    (x, ok), used = device_bytes_during(
        lambda: gpu.linear_solve(ptr, idx, val, rhs, fp32_matrix=True))
    assert ok
    val = val.astype(np.float32).astype(np.float64)
    residual = rhs - np.add.reduceat(val * x[idx], ptr[:-1])
    assert np.linalg.norm(residual) <= 2e-6 * (1 + np.linalg.norm(rhs))
    # entries, the 128 MB, a dozen vectors, and 48 MB for what else the driver takes
    bound = 12 * ptr[-1] + (128 << 20) + 12 * 8 * n + (48 << 20)
    assert 12 * ptr[-1] < used <= bound, (used, bound)


@pytest.mark.parametrize("kept", [1, 3])
def test_compaction_memory(gpu, kept):
    """The device holds the source and the entries that are kept, not room for all that
    could be: 40 M entries, of which a few columns keep 1 in 1,000 (an output inside
    the call's one allocation would take 640 MB more) or 3 in 4."""
    rows, per, n = 400_000, 100, 1000
    rng = np.random.default_rng(18)
    idx = np.sort(rng.integers(0, n, (rows, per)), axis=1).reshape(-1)
    val = rng.standard_normal(idx.size)
    ptr = per * np.arange(rows + 1, dtype=np.int64)
    stay = np.zeros(n, dtype=bool)
    stay[500 if kept == 1 else np.arange(n) % 4 != 0] = True
    cmap = np.where(stay, np.cumsum(stay) - 1, -1)
    gpu.compact_csr(ptr[:2], idx[:per], val[:per], n, [0], cmap, int(stay.sum()))
    (p, i, v), used = device_bytes_during(
        lambda: gpu.compact_csr(ptr, idx, val, n, np.arange(rows), cmap, int(stay.sum())))
    take = stay[idx]
    assert np.array_equal(i, cmap[idx[take]]) and np.array_equal(v, val[take])
    assert np.array_equal(p, np.r_[0, np.cumsum(take.reshape(rows, per).sum(axis=1))])
    bound = 16 * (idx.size + i.size) + 8 * (5 * rows + n) + (48 << 20)
    assert 16 * idx.size < used <= bound, (used, bound)


@pytest.mark.parametrize("lens", [[5000], [0] * 31 + [1281], [640, 0, 1, 639, 3], [20] * 31 + [21],
                                  [700] * 33, [1] * 32 + [640] * 2 + [5] * 40])
def test_propagate_bounds_long_groups(gpu, oracle, lens):
    """Groups of 32 rows with more than the 640 entries that a warp holds at a time: one
    long row, rows that end at and cross its edges, a single entry more; bit-identical
    to the sequential restatement."""
    rng = np.random.default_rng(19)
    n = sum(lens)
    cols = np.split(rng.permutation(n), np.cumsum(lens)[:-1])
    m = tiny(n, len(lens), [(i, int(j), float(v)) for i, js in enumerate(cols)
                            for j, v in zip(np.sort(js), np.round(rng.standard_normal(js.size), 1))])
    lb, ub = rng.uniform(-5, 0, n), rng.uniform(0, 40, n)
    # rows held near their greatest activity, so that most columns are tightened; where
    # there are several rows, one column of the last without an upper bound
    row = np.repeat(np.arange(m.m), np.diff(m.ptr))
    high = np.bincount(row, weights=np.maximum(m.val * lb[m.idx], m.val * ub[m.idx]),
                       minlength=m.m)
    m.rl, m.ru = high - rng.uniform(0.5, 3, m.m), np.full(m.m, np.inf)
    if np.count_nonzero(lens) > 1:
        ub[m.idx[-1]] = np.inf
    integer = (np.arange(n) % 3 == 0).astype(np.int32)
    got = gpu.propagate_bounds(m, integer, lb, ub, 4)
    want = oracle.propagate_bounds(m, integer, lb, ub, 4)
    assert got[0] == want[0]
    assert np.sum((want[1] != lb) | (want[2] != ub)) >= n // 3
    for u, w in zip(got[1:], want[1:]):
        assert np.array_equal(u.view(np.int64), w.view(np.int64))


@pytest.mark.parametrize("n,band,resident", [(600, 23, True), (600, 25, True), (2001, 2001, True),
                                             (240_001, 3, False), (240_001, 27, False),
                                             (3001, 3001, False)])
def test_sparse_q_paths(gpu, oracle, n, band, resident):
    """A sparse Q's rows walked in the primal kernel (24 entries or fewer on average) and
    shared by lanes (more), in models whose trials run in one launch and, with a large Q
    or a large A, as kernels of their own: the same bits either way, and the oracle's
    sequential row sums to rounding (rows of up to 3,001 terms of one size, 7e-13 a
    trial)."""
    m = synth.random_lp(m=n // 2, n=n, per_col=5, seed=20)
    i, half = np.arange(n), band // 2
    rows = np.repeat(i, 2 * half + 1)
    cols = (rows + np.tile(np.arange(-half, half + 1), n)) % n
    vals = np.where(rows == cols, 1.0, -0.5 / band)
    order = np.lexsort((cols, rows))
    m.qptr = (2 * half + 1) * np.arange(n + 1, dtype=np.int64)
    m.qidx, m.qval = cols[order].astype(np.int64), vals[order]
    tau, sigma = (0.3 * v for v in step_sizes(m))
    a, b = (gpu.PdhgBackend(m, graphs=True) for _ in range(2))
    info = a.layout_info()
    assert info["resident"] == resident, info
    assert info["kernels_per_trial"] == (2 if band <= 24 else 3), info
    cpu = oracle.model(m).backend(np.zeros(m.n), np.zeros(m.m))
    # the step sizes that advance() reduces a QP's own to
    ptr = np.r_[0, np.cumsum(np.abs(m.val))]
    norm = math.sqrt(np.max(ptr[m.ptr[1:]] - ptr[m.ptr[:-1]])) * math.sqrt(
        np.bincount(m.idx, weights=np.abs(m.val), minlength=n).max())
    scale = min(1.0, 0.9 / (math.sqrt(tau * sigma) * norm + tau * 1.6))
    assert scale == 1.0
    for count in (1, 9):
        a.advance(count, tau, sigma)
        b.profile_kernels(count, tau, sigma)
        cpu.advance(count, tau, sigma)
        for u, w, z in zip(a.candidates(), b.candidates(), cpu.candidates()):
            assert np.array_equal(u, w)
            near(u, z)


@pytest.mark.parametrize("method", ["adaptive", "halpern", "sparse q"])
def test_resident_and_kernel_trials_alternate(gpu, method):
    """With several engines in flight a call's trials may run as kernels of their own
    and the next call's in one launch: an engine that alternates ends, bit for bit,
    where one that never runs resident does."""
    m = synth.random_lp(m=900, n=2001, per_col=5, seed=21)
    if method == "sparse q":
        m.qptr, m.qidx, m.qval = sparse_q(m.n, "low rank")
    # the step sizes that advance() would reduce a QP's own to are below its limit
    tau, sigma = (v * (0.01 if method == "sparse q" else 1) for v in step_sizes(m))
    options = dict(adaptive=method == "adaptive", halpern=method == "halpern", graphs=True)
    if method == "halpern":
        options.update(reflection=0.5, residual_restarts=True)
    a, b = gpu.PdhgBackend(m, **options), gpu.PdhgBackend(m, **options)
    assert a.layout_info()["resident"]
    for k, count in enumerate((3, 7, 30, 2, 1, 40, 5)):
        (a.profile_kernels if k % 2 else a.advance)(count, tau, sigma)
        b.profile_kernels(count, tau, sigma)
        for u, w in zip(a.candidates(), b.candidates()):
            assert np.array_equal(u, w)
        if a.restart_requested():
            for g in (a, b):
                g.reset_candidate(True)
    assert a.rejected_steps() == b.rejected_steps()


def test_many_engines_in_flight(gpu):
    """Eight engines from eight threads, more than run resident at once: each ends where
    it ends alone, bit for bit."""
    import threading
    models = [synth.random_lp(m=m, n=2 * m + 1, per_col=4, seed=m) for m in
              (400, 9000, 2000, 20000, 500, 3000, 12000, 5000)]
    steps = [step_sizes(m) for m in models]

    def run(k, out):
        g = gpu.PdhgBackend(models[k], adaptive=k % 2 == 0, halpern=k % 2 == 1, graphs=True)
        for _ in range(25):
            g.advance(40, *steps[k])
        out[k] = g.candidates()

    alone, together = {}, {}
    for k in range(8):
        run(k, alone)
    threads = [threading.Thread(target=run, args=(k, together)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(8):
        for u, w in zip(alone[k], together[k]):
            assert np.array_equal(u, w)


def test_walked_sparse_q_memory(gpu):
    """A sparse Q walked in the primal kernel takes its own storage and nothing else."""
    m = synth.random_lp(m=20_000, n=40_001, per_col=5, seed=22)
    lp = gpu.PdhgBackend(m, indices="64").stats()["device_bytes"]
    i = np.arange(m.n)
    rows = np.repeat(i, 3)
    cols = np.sort(np.stack([(i - 1) % m.n, i, (i + 1) % m.n], axis=1), axis=1).reshape(-1)
    m.qptr, m.qidx = 3 * np.arange(m.n + 1, dtype=np.int64), cols.astype(np.int64)
    m.qval = np.where(rows == cols, 2.0, -1.0)
    qp = gpu.PdhgBackend(m, indices="64").stats()["device_bytes"]
    assert 16 * cols.size < qp - lp <= 16 * cols.size + 8 * (m.n + 1) + 4 * m.n + 4096
