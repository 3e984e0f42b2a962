"""Octrees and treecode evaluations at the sizes where the point sort changes its path: registers per thread of the
one-cluster sort, the many-block passes above it, the pair sort of deep trees; exact against the oracle's trees."""
import numpy as np
import pytest

import lpmcxx_b200 as L
import oracle

pytestmark = pytest.mark.gpu

BOX = (-1.00001, 1.00001) * 3


def _points(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    x[: n // 2] = x[: n // 2] * 0.02 + (0.5, -0.3, 0.2)  # half of them clustered: deep, uneven nodes
    x /= np.maximum(1.0, np.abs(x).max(axis=1, keepdims=True) * 1.001)
    return oracle.pack4(x)


def _check(tree, ref):
    members, offsets = tree.leaf_membership()
    assert np.array_equal(offsets, ref["leaf_offsets"]) and np.array_equal(members, ref["members"])
    nodes = tree.nodes()
    for k in ("node_level", "node_parent", "node_count", "node_box"):
        assert np.array_equal(nodes[k], ref[k])


@pytest.mark.parametrize("n", [1, 31, 33, 8191, 32768, 32769, 65536, 65537, 131071, 131072, 131073, 300001])
@pytest.mark.parametrize("depth", [10, 21])
def test_tree_at_sort_boundaries(ctx, n, depth):
    torch = ctx.use_torch_stream()
    pts = _points(n, n)
    ref = oracle.tree_build(pts, BOX, 40, depth)
    tree = L.Tree(ctx, torch.tensor(pts, device="cuda"), BOX, 40, depth, allow_overflow=True)
    _check(tree, ref)
    tree.close()


@pytest.mark.parametrize("n", [1, 127, 129, 4097, 65537, 131072, 131073])
def test_poisson_treecode_at_batch_cut_boundaries(ctx, n):
    """theta so small that every pair is near: the treecode is then its FP32 direct sum (5e-6 as the FP32 parity
    tests), and a batch cut or list offset that loses or repeats a target or a range shows at once."""
    torch = ctx.use_torch_stream()
    rng = np.random.default_rng(n)
    d = torch.tensor(rng.uniform(-1, 1, (n, 4)), device="cuda")
    ts = L.TreeSum(ctx, L.poisson_kernel(), L.tree_solver(L.LPM_PREC_F32, 4, 200, 1e-6), n, n)
    out = torch.full((1, n), float("nan"), dtype=torch.float64, device="cuda")
    ref = torch.empty_like(out)
    ctx.direct_sum_dev(L.poisson_kernel(), L.LPM_PREC_F64, d, d, ref, n)
    for _ in range(2):
        ts.eval(d, d, out)
        assert torch.isfinite(out).all()
        assert float((out - ref).norm()) <= 5e-6 * float(ref.norm())
    ts.close()


@pytest.mark.parametrize("n,depth", [(65536, 21), (65537, 21), (524288, 10), (524289, 10), (700001, 21)])
def test_tree_at_digit_scan_boundaries(ctx, n, depth):
    """The digit counts of a many-block pass, 256 per 4096 keys, scanned by a block (65,536 pairs), by a cluster with one
    run of 128 a warp (up to 524,288 keys) and with several."""
    torch = ctx.use_torch_stream()
    pts = _points(n, n)
    tree = L.Tree(ctx, torch.tensor(pts, device="cuda"), BOX, 200, depth, allow_overflow=True)
    _check(tree, oracle.tree_build(pts, BOX, 200, depth))
    tree.close()
