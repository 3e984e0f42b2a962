"""Treecode evaluations whose batches run on clusters of blocks (few batches): the same stages and tiles, so the result of
one block per batch up to the order of its FP64 additions."""
import numpy as np
import pytest

import lpmcxx_b200 as L
import lpmcxx_b200.workloads as W

pytestmark = pytest.mark.gpu


def _fibonacci(n, seed):
    i = np.arange(n) + 0.5
    z = 1.0 - 2.0 * i / n
    phi = np.pi * (1.0 + 5.0 ** 0.5) * i
    r = np.sqrt(1.0 - z * z)
    q, _ = np.linalg.qr(np.random.default_rng(seed).normal(size=(3, 3)))
    return np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1) @ q


@pytest.mark.parametrize("n", [300, 9000, 30011, 60000, 140000])
@pytest.mark.parametrize("solver", [dict(order=1, theta=0.4), dict(order=8, theta=0.6), dict(order=10, learned=True, theta=0.5)])
def test_ensemble_of_one_equals_cluster_launches(ctx, n, solver):
    """An ensemble's instance sums every batch in one block, an RK4 of its own on clusters: one step from the same
    state, compared at 1e-14 (dt times the FP64 rounding of a velocity of order 1)."""
    rng = np.random.default_rng(n)
    state = np.zeros((n, 4))
    state[:, :3] = _fibonacci(n, n)
    n_src = 2 * n // 3
    state[:n_src, 3] = W.gaussian_vortex(state[:n_src, :3], np.array([0.0, 0.6, 0.8])) / n + rng.normal(size=n_src) / n ** 1.5
    desc = L.tree_solver(L.LPM_PREC_F32, max_per_leaf=128, tolerance=5e-7 if "learned" in solver else 0.0, **solver)
    params = L.learned.load()[0] if "learned" in solver else None
    kernel = L.biot_savart_kernel()
    ens = L.Ensemble(ctx, kernel, desc, [n_src], [n], lanes=1)
    rk = L.RK4(ctx, kernel, desc, n_src, n)
    if params is not None:
        ens.set_mlp(params)
        rk.set_mlp(params)
    ens.instance(0).set_state(state)
    rk.set_state(state)
    ens.step(0.01, 2, use_graph=True)
    rk.step(0.01, 2, use_graph=True)
    a, b = ens.instance(0).get_state(), rk.get_state()
    ens.close()
    rk.close()
    assert np.abs(a - state).max() > 1e-6
    assert np.abs(a - b).max() < 1e-14


@pytest.mark.parametrize("n", [400, 20000, 100000])
@pytest.mark.parametrize("order", [0, 6, 11])
def test_poisson_clusters_against_direct(ctx, n, order):
    """Wide acceptance at order 6 and 11, none worth an expansion at order 0: within the truncation the unsplit
    launches have at these orders (1e-3, 1e-4; 5e-6 where every pair is summed directly), every target written."""
    torch = ctx.use_torch_stream()
    rng = np.random.default_rng(n + order)
    d = torch.tensor(rng.uniform(-1, 1, (n, 4)), device="cuda")
    theta = {0: 1e-6, 6: 0.6, 11: 0.5}[order]
    ts = L.TreeSum(ctx, L.poisson_kernel(), L.tree_solver(L.LPM_PREC_F32, order, 200, theta), n, n)
    out = torch.full((1, n), float("nan"), dtype=torch.float64, device="cuda")
    ref = torch.empty_like(out)
    ctx.direct_sum_dev(L.poisson_kernel(), L.LPM_PREC_F64, d, d, ref, n)
    ts.eval(d, d, out)
    ts.close()
    assert float((out - ref).norm()) <= {0: 5e-6, 6: 1e-3, 11: 1e-4}[order] * float(ref.norm())
