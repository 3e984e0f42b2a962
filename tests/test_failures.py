"""Failure paths, injected on the host: non-finite input, a device allocation that fails (through the
library's injection point, lpm_debug_fail_allocations), and a capacity overflow inside a captured RK4 replay.
Each reports its status code, and the context stays usable afterwards.  No GPU fault is caused."""
import numpy as np
import pytest

import lpmcxx_b200 as L
import lpmcxx_b200.workloads as W


@pytest.mark.gpu
def test_nan_source_is_reported(ctx):
    """A non-finite source coordinate makes the treecode's root box non-finite: the evaluation fails with
    LPM_ERR_ARG (no result is written from an incomplete tree), and the next valid evaluation succeeds."""
    torch = ctx.use_torch_stream()
    _, p, n_src = W.gaussian_vortex_mesh("icos", 4)
    bad = p.copy()
    bad[7, 0] = np.nan
    ts = L.TreeSum(ctx, L.biot_savart_kernel(), L.tree_solver(L.LPM_PREC_F32, 8, 64, 0.5), n_src, p.shape[0])
    out = torch.empty((3, p.shape[0]), dtype=torch.float64, device="cuda")
    d_bad = torch.tensor(bad, device="cuda")
    with pytest.raises(L.LpmError) as e:
        ts.eval(d_bad[:n_src], d_bad, out)
    assert e.value.code == L._capi.LPM_ERR_ARG
    d = torch.tensor(p, device="cuda")
    ts.eval(d[:n_src], d, out)
    assert torch.isfinite(out).all()
    ts.close()


@pytest.mark.gpu
def test_injected_allocation_failure_reports_oom_and_recovers(ctx):
    """Every device allocation of solver creation and of the first evaluation, failed in turn: the entry
    point that made it returns LPM_ERR_OOM (nothing leaks into later calls), and with the injection off the
    same calls succeed and agree with an undisturbed run."""
    torch = ctx.use_torch_stream()
    _, p, n_src = W.gaussian_vortex_mesh("icos", 4)
    d = torch.tensor(p, device="cuda")
    solver = L.tree_solver(L.LPM_PREC_F32, 8, 64, 0.5)
    want = torch.empty((3, p.shape[0]), dtype=torch.float64, device="cuda")
    ts = L.TreeSum(ctx, L.biot_savart_kernel(), solver, n_src, p.shape[0])
    ts.eval(d[:n_src], d, want)
    ts.close()
    failed = 0
    lib = L.lib()
    try:
        for k in range(60):
            lib.lpm_debug_fail_allocations(k)
            try:
                ts = L.TreeSum(ctx, L.biot_savart_kernel(), solver, n_src, p.shape[0])
                out = torch.empty_like(want)
                ts.eval(d[:n_src], d, out)
                ts.close()
            except L.LpmError as e:
                assert e.code == L._capi.LPM_ERR_OOM, (k, e)
                failed += 1
                continue
            break  # k passed every allocation of creation and evaluation
    finally:
        lib.lpm_debug_fail_allocations(-1)
    assert failed > 5
    ts = L.TreeSum(ctx, L.biot_savart_kernel(), solver, n_src, p.shape[0])
    out = torch.empty_like(want)
    ts.eval(d[:n_src], d, out)
    ts.close()
    assert torch.equal(out, want)


@pytest.mark.gpu
def test_capacity_overflow_in_captured_replay_is_reported_and_recovers(ctx):
    """An RK4 step graph captured while every particle sits in one octree cell (a step of 1e-12 moves them by
    1e-7, inside the cell) holds interaction lists sized for that state; replayed on the spread-out mesh it needs
    ~8x more near-field entries than it holds: the step reports LPM_ERR_CAPACITY instead of returning wrong
    velocities.  An uncaptured step then regrows the lists, and the next graph step with the same dt captures a
    new graph (the old one holds the freed lists' addresses) whose result equals the uncaptured step's."""
    _, p, n_src = W.gaussian_vortex_mesh("icos", 5)
    tiny = p.copy()
    x0 = np.array([0.0, 0.0, 1.0])
    tiny[:, :3] = x0 + 1e-9 * (p[:, :3] - x0)
    tiny[:, :3] /= np.linalg.norm(tiny[:, :3], axis=1, keepdims=True)
    dt = 1e-12
    rk = L.RK4(ctx, L.biot_savart_kernel(), L.tree_solver(L.LPM_PREC_F32, 4, 1, 0.3), n_src, p.shape[0])
    rk.set_state(tiny)
    rk.step(dt, 2, use_graph=True)  # one uncaptured step sizes the lists, then one graph replay
    rk.set_state(p)
    with pytest.raises(L.LpmError) as e:
        rk.step(dt, 1, use_graph=True)
    assert e.value.code == L._capi.LPM_ERR_CAPACITY
    rk.set_state(p)
    rk.step(dt, 1, use_graph=False)  # regrows the lists
    want = rk.get_state()
    rk.set_state(p)
    rk.step(dt, 1, use_graph=True)  # same dt: captured again because the lists moved
    got = rk.get_state()
    rk.close()
    assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("scalar", [False, True])
def test_failed_regrow_leaves_the_solver_usable(ctx, scalar):
    """One solver, sized by an evaluation of particles that sit in one octree cell: each allocation of the regrow that
    the spread-out particles then need fails in turn.  The call returns LPM_ERR_OOM, at least one of the buffers that
    went is counted as empty (so that no kernel writes where nothing is), and both inputs evaluate afterwards as on a
    fresh solver."""
    torch = ctx.use_torch_stream()
    _, p, n_src = W.gaussian_vortex_mesh("icos", 5)
    tiny = p.copy()
    x0 = np.array([0.0, 0.0, 1.0])
    tiny[:, :3] = x0 + 1e-9 * (p[:, :3] - x0)
    tiny[:, :3] /= np.linalg.norm(tiny[:, :3], axis=1, keepdims=True)
    kernel = L.poisson_kernel() if scalar else L.biot_savart_kernel()
    solver = L.tree_solver(L.LPM_PREC_F32, 4, 4, 0.3)
    inputs = [torch.tensor(a, device="cuda") for a in (tiny, p)]
    comps = 1 if scalar else 3

    def evaluate(ts, d):
        out = torch.full((comps, p.shape[0]), float("nan"), dtype=torch.float64, device="cuda")
        ts.eval(d[:n_src], d, out)
        return out

    want = []
    for d in inputs:
        fresh = L.TreeSum(ctx, kernel, solver, n_src, p.shape[0])
        want.append(evaluate(fresh, d))
        fresh.close()
    lib, failed = L.lib(), 0
    for k in range(20):
        ts = L.TreeSum(ctx, kernel, solver, n_src, p.shape[0])
        evaluate(ts, inputs[0])
        try:
            lib.lpm_debug_fail_allocations(k)
            evaluate(ts, inputs[1])
            done = True
        except L.LpmError as e:
            assert e.code == L._capi.LPM_ERR_OOM, (k, e)
            done = False
        finally:
            lib.lpm_debug_fail_allocations(-1)
        if not done:
            assert 0 in [ts.get_param(c) for c in ("far_cap", "near_cap", "heavy_cap")]
            failed += 1
        for i in (0, 1, 0):
            assert torch.equal(evaluate(ts, inputs[i]), want[i]), (k, i)
        ts.close()
        if done:
            break
    assert done and failed >= 2


@pytest.mark.gpu
@pytest.mark.parametrize("n", [110000, 200000])
def test_more_batches_than_the_capacity_are_reported(ctx, n):
    """Targets that fill a volume occupy 8^4 cells of the finest batch level, where the capacity is made for the cells
    that a sphere meets: LPM_ERR_CAPACITY, with no more batches in use than the arrays hold (one launch cuts the batches
    up to 131,072 targets, several above).  The level below fits, and the solver evaluates on it."""
    torch = ctx.use_torch_stream()
    rng = np.random.default_rng(n)
    tgt = torch.tensor(rng.uniform(-1, 1, (n, 4)), device="cuda")
    src = tgt[:1000].clone()
    ts = L.TreeSum(ctx, L.biot_savart_kernel(), L.tree_solver(L.LPM_PREC_F32, 4, 64, 0.5), 1000, n)
    ts.set_param("root_maxr", 1.0)
    assert ts.get_param("batch_level_max") == 4 and ts.get_param("batch_cap") < 8 ** 4
    out = torch.empty((3, n), dtype=torch.float64, device="cuda")
    ts.set_param("batch_level", 4)
    for _ in range(2):
        with pytest.raises(L.LpmError, match="4096 target batches") as e:
            ts.eval(src, tgt, out)
        assert e.value.code == L._capi.LPM_ERR_CAPACITY
        assert ts.stats()["batches"] == ts.get_param("batch_cap")
    ts.set_param("batch_level", 3)
    ts.eval(src, tgt, out)
    assert ts.stats()["batches"] < ts.get_param("batch_cap")
    ts.close()


@pytest.mark.gpu
def test_output_over_the_targets_survives_a_regrow(ctx):
    """out may lie over the targets' storage (they are read before it is written), also where the evaluation needs larger
    buffers than an earlier one left: it is then not repeated on inputs that its first pass has overwritten."""
    torch = ctx.use_torch_stream()
    _, p, n_src = W.gaussian_vortex_mesh("icos", 5)
    tiny = p.copy()
    x0 = np.array([0.0, 0.0, 1.0])
    tiny[:, :3] = x0 + 1e-9 * (p[:, :3] - x0)
    tiny[:, :3] /= np.linalg.norm(tiny[:, :3], axis=1, keepdims=True)
    n = p.shape[0]
    small, d = torch.tensor(tiny, device="cuda"), torch.tensor(p, device="cuda")
    src, want = d[:n_src].clone(), torch.empty((3, n), dtype=torch.float64, device="cuda")
    results = []
    for alias in (False, True):
        ts = L.TreeSum(ctx, L.biot_savart_kernel(), L.tree_solver(L.LPM_PREC_F32, 4, 1, 0.3), n_src, n)
        ts.eval(small[:n_src], small, want)
        held = ts.get_param("near_cap")
        out = d.view(-1)[: 3 * n].view(3, n) if alias else want
        ts.eval(src, d, out)
        assert ts.get_param("near_cap") > held
        results.append(out.clone())
        ts.close()
    assert torch.equal(*results)
