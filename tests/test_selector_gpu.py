"""The order selector at the edges of its tiles and of the traversal's decision cache."""
import numpy as np
import pytest

import lpmcxx_b200 as L
from lpmcxx_b200 import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,theta", [(8, 0.05), (200, 0.3)])
def test_more_decisions_than_the_cache_holds(ctx, leaf, theta):
    """Leaves of 8 sources and a narrow acceptance put more than 1024 accepted clusters on a batch (leaves of 200 far
    fewer); the fill pass then selects again, and a decision other than the count pass's shifts or drops entries.
    Budget 1e-9 of sum|w| a pair, up to 1e4 pairs, velocities of about 0.1 sum|w| / 4 pi: 1e-4, and 5e-6 for FP32."""
    torch = ctx.use_torch_stream()
    n = 40000
    rng = np.random.default_rng(leaf)
    x = rng.normal(size=(n, 3))
    state = np.zeros((n, 4))
    state[:, :3] = x / np.linalg.norm(x, axis=1, keepdims=True)
    state[:, 3] = rng.uniform(0.5, 1.5, n) * (1.0 + state[:, 2]) / n
    desc = L.tree_solver(L.LPM_PREC_F32, order=10, learned=True, theta=theta, max_per_leaf=leaf, tolerance=1e-9)
    rk = L.RK4(ctx, L.biot_savart_kernel(), desc, n, n)
    rk.set_mlp(learned.load()[0])
    rk.set_state(state)
    out = torch.full((3, n), float("nan"), dtype=torch.float64, device="cuda")
    rk.velocity(out)
    stats = rk.tree_stats()
    rk.close()
    d = torch.tensor(state, device="cuda")
    ref = torch.empty_like(out)
    ctx.direct_sum_dev(L.biot_savart_kernel(), L.LPM_PREC_F64, d, d, ref, n)
    entries = (stats["far_pairs"] + stats["near_runs"]) / stats["batches"]
    assert (entries > 2048) == (leaf == 8)
    assert stats["overflow"] == 0
    assert float((out - ref).norm()) <= 1.05e-4 * float(ref.norm())


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 1000])
def test_classes_at_tile_edges(ctx, n):
    """A sample's class does not depend on the rows beside it: the first n of 1024 samples on their own."""
    params = learned.load()[0]
    f = np.random.default_rng(5).normal(size=(1024, 8)).astype(np.float32) * 2.0
    assert np.array_equal(L.mlp_predict(ctx, params, f[:n]), L.mlp_predict(ctx, params, f)[:n])


@pytest.mark.parametrize("n", [1, 127, 129, 75775, 75777, 151553])
def test_predictions_do_not_depend_on_the_grid(ctx, n):
    """One launch of at most four blocks per SM, whose warps take 32 samples at a time: the classes of n samples are those
    of their runs of 1,000 samples (no warp takes more than 32 there)."""
    params = learned.load()[0]
    feats = np.random.default_rng(n).normal(size=(n, 8)).astype(np.float32)
    got = L.mlp_predict(ctx, params, feats)
    runs = [L.mlp_predict(ctx, params, feats[i:i + 1000]) for i in range(0, n, 1000)]
    assert np.array_equal(got, np.concatenate(runs))
