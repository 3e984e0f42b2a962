"""Direct sums at the sizes where their source splits change: thread groups, cluster parts, ragged tiles and targets.

Tolerances.  FP64: each of the at most n_src terms and their sum round within 2^-53 of sum |terms|, and a close pair's
denominator within 2^-53 / den, 2e-12 of the pair at the closest spacing here; against the largest component 1e-12 (as
the other FP64 parity tests).  FP32: 5e-6 relative L2 (as the other FP32 tests).  Sums that differ only in the order of
their FP64 additions: 1e-13.
"""
import numpy as np
import pytest

import lpmcxx_b200 as L
import oracle
from conftest import rel_l2, rel_linf
from test_direct_sum_gpu import random_sphere

pytestmark = pytest.mark.gpu

SIZES = [(2, 1), (63, 129), (64, 128), (127, 511), (512, 513), (513, 31), (1025, 1025), (2049, 4735), (5121, 7777),
         (16385, 300), (300, 60001)]


def _data(n_src, n_tgt, scalar):
    rng = np.random.default_rng(n_src + 3 * n_tgt)
    n = max(n_src, n_tgt)
    pts = rng.uniform(-1.0, 1.0, (n, 3)) if scalar else random_sphere(n, n)
    src = oracle.pack4(pts[:n_src], rng.uniform(-1, 1, n_src) / n_src)
    return src, oracle.pack4(pts[:n_tgt])


def _sum(ctx, kernel, prec, src, tgt, comps, coinc):
    import torch

    out = torch.full((comps, tgt.shape[0]), float("nan"), dtype=torch.float64, device="cuda")
    ctx.direct_sum_dev(kernel, prec, torch.tensor(src, device="cuda"), torch.tensor(tgt, device="cuda"), out, coinc)
    return out.cpu().numpy()


@pytest.mark.parametrize("n_src,n_tgt", SIZES)
@pytest.mark.parametrize("delta", [0.0, 0.03])
def test_biot_savart_split(ctx, n_src, n_tgt, delta):
    ctx.use_torch_stream()
    src, tgt = _data(n_src, n_tgt, False)
    kernel, coinc = L.biot_savart_kernel(1.0, delta), min(n_src, n_tgt)
    ref = oracle.bs_direct(src, tgt, delta=delta)
    got = _sum(ctx, kernel, L.LPM_PREC_F64, src, tgt, 3, coinc)
    assert rel_linf(got, ref) < 1e-12
    if not np.any(ref):
        return
    first = None
    for targets in (2, 4, 8):
        ctx.set_param("direct_targets", targets)
        f32 = _sum(ctx, kernel, L.LPM_PREC_F32, src, tgt, 3, coinc)
        ctx.set_param("direct_targets", 4)
        assert rel_l2(f32, ref) < 5e-6
        first = f32 if first is None else first
        assert rel_linf(f32, first) < 1e-13


@pytest.mark.parametrize("n_src,n_tgt", SIZES)
def test_poisson_split(ctx, n_src, n_tgt):
    ctx.use_torch_stream()
    src, tgt = _data(n_src, n_tgt, True)
    ref = oracle.poisson_direct(src, tgt)
    got = _sum(ctx, L.poisson_kernel(), L.LPM_PREC_F64, src, tgt, 1, min(n_src, n_tgt))[0]
    assert rel_linf(got, ref) < 1e-12
    f32 = _sum(ctx, L.poisson_kernel(), L.LPM_PREC_F32, src, tgt, 1, min(n_src, n_tgt))[0]
    if np.any(ref):
        assert rel_l2(f32, ref) < 5e-6


def test_reciprocals_to_the_last_bits(ctx):
    """One pair per target (the other sources have strength 0): r (1 + e + e^2) and y (1 + e (1/2 + 3/8 e)) against
    80-bit results.  Biot-Savart: three roundings of den (3 2^-53 / den), five more of the product and cross product."""
    ctx.use_torch_stream()
    n = 4001
    t = np.linspace(0.06, np.pi, n)
    tgt = oracle.pack4(np.stack([np.cos(t), np.sin(t), np.zeros(n)], axis=1))
    src = oracle.pack4(np.tile([0.0, 0.0, 1.0], (300, 1)))
    src[100] = (1.0, 0.0, 0.0, 1.0)
    got = _sum(ctx, L.biot_savart_kernel(), L.LPM_PREC_F64, src, tgt, 3, 0)[2]
    x = tgt.astype(np.longdouble)
    den = 1 - x[:, 0]
    ref = x[:, 1] / den / (4 * np.longdouble(np.pi))  # -(x cross y)_z / (4 pi den), y = (1, 0, 0)
    assert np.max(np.abs(got / ref - 1) / (2.0 ** -53 * (8 + 3 / den))) < 1.0
    phi = _sum(ctx, L.poisson_kernel(), L.LPM_PREC_F64, src, tgt, 1, 0)[0]
    r = np.sqrt((x[:, 0] - 1) ** 2 + x[:, 1] ** 2)
    assert np.max(np.abs(phi * (4 * np.longdouble(np.pi)) * r - 1)) < 8 * 2.0 ** -53


def test_values_that_are_not_finite(ctx):
    """A NaN coordinate spoils the components it enters and no others, as the reference's expression does."""
    ctx.use_torch_stream()
    src, tgt = _data(700, 300, False)
    src[400, 0] = np.nan
    got = _sum(ctx, L.biot_savart_kernel(), L.LPM_PREC_F64, src, tgt, 3, 0)
    assert np.isfinite(got[0]).all() and np.isnan(got[1:]).all()
    tgt2 = tgt.copy()
    tgt2[7, :3] = np.nan
    clean, _ = _data(700, 300, False)
    got = _sum(ctx, L.biot_savart_kernel(), L.LPM_PREC_F64, clean, tgt2, 3, 0)
    assert np.isnan(got[:, 7]).all() and np.isfinite(np.delete(got, 7, axis=1)).all()
    phi = _sum(ctx, L.poisson_kernel(), L.LPM_PREC_F64, src, tgt, 1, 0)[0]
    assert rel_linf(phi, oracle.poisson_direct(np.delete(src, 400, axis=0), tgt)) < 1e-12


@pytest.mark.parametrize("kernel", [L.sphere_greens_kernel(), L.planar_log_kernel()])
@pytest.mark.parametrize("scale", [1.0, 3e-60, 7e70])
def test_log_kernels_to_the_last_bits(ctx, kernel, scale):
    """One pair per target (the other sources have strength 0), arguments of the logarithm from 2^-9 to 2 (sphere) and
    over many binades and about 1 (plane), against 80-bit logarithms: 2 units of the last place of the logarithm's two
    summands (k log 2 and the rest, each below |log| + 0.7), and the sphere's fused argument 3 2^-53 / z."""
    sphere = kernel.kind == L.sphere_greens_kernel().kind
    if sphere and scale != 1.0:
        pytest.skip("the sphere kernel's points have its radius")
    ctx.use_torch_stream()
    n = 6001
    if sphere:
        t = np.linspace(0.07, np.pi, n)
        tgt = oracle.pack4(np.stack([np.cos(t), np.sin(t), np.zeros(n)], axis=1))
    else:
        r = np.concatenate([np.exp(np.linspace(-12, 12, n - 2001)), 1.0 + np.linspace(-0.02, 0.02, 2001)])
        tgt = oracle.pack4(np.stack([1.0 + r, np.zeros(n), np.zeros(n)], axis=1) * scale)
    src = oracle.pack4(np.tile([0.0, 0.0, 1.0], (300, 1)) * scale)
    src[100] = (scale, 0.0, 0.0, 1.0)
    got = _sum(ctx, kernel, L.LPM_PREC_F64, src, tgt, 1, 0)[0]
    x = tgt.astype(np.longdouble)
    if sphere:
        z = 1 - x[:, 0]
        ref, cond = -np.log(z) / (4 * np.longdouble(np.pi)), 3 / z
    else:
        d = (x[:, 0] - np.longdouble(src[100, 0]))
        dr = (tgt[:, 0] - src[100, 0]).astype(np.longdouble)  # x - y rounds once in FP64
        z, cond = dr * dr, np.abs(2 * (d - dr) / dr) * 2.0 ** 53 + 1
        ref = np.log(z) / (4 * np.longdouble(np.pi))
    tol = 2.0 ** -53 * (2 * (2 * np.abs(np.log(z)) + 0.7) + cond) / (4 * np.pi)
    assert np.max(np.abs(got - ref) / tol) < 1.0


@pytest.mark.parametrize("kernel,comps", [(L.biot_savart_kernel(), 3), (L.biot_savart_kernel(1.0, 0.03), 3),
                                          (L.sphere_greens_kernel(), 1), (L.poisson_kernel(), 1)])
def test_targets_missing_from_a_block_change_nothing(ctx, kernel, comps):
    """Targets far from every source (none takes the path of close pairs) have the same sums, bit for bit, in a full block
    of 64 as in one that holds only them: what stands in for missing targets sends no warp down another path."""
    ctx.use_torch_stream()
    x = random_sphere(3000, 3)
    north, south = x[x[:, 2] > 0.3][:700], x[x[:, 2] < -0.2][:64]
    src, tgt = oracle.pack4(north, np.linspace(-1.0, 1.0, 700)), oracle.pack4(south)
    full = _sum(ctx, kernel, L.LPM_PREC_F64, src, tgt, comps, 0)
    for n in (1, 2, 33, 63):
        assert np.array_equal(_sum(ctx, kernel, L.LPM_PREC_F64, src, tgt[:n], comps, 0), full[:, :n]), n


@pytest.mark.parametrize("n_src,n_tgt", [(0, 20721), (1, 20719), (1, 20721), (2, 30001), (127, 147999), (128, 148001),
                                         (129, 148001), (257, 75003), (511, 75003), (513, 113667), (1025, 75003)])
@pytest.mark.parametrize("name", ["bs", "bs_delta", "poisson", "greens", "log", "delta3d", "sphere_delta"])
def test_few_sources_many_targets(ctx, name, n_src, n_tgt):
    """Around the targets per SM from which up to 128 sources take the kernel without splits, and around the sources from
    which crowded SMs get parts; the reference on the first, the last and every 37th target."""
    ctx.use_torch_stream()
    make, kind, param = {"bs": (L.biot_savart_kernel, 1, 0.0), "bs_delta": (L.biot_savart_kernel, 1, 0.03),
                         "poisson": (L.poisson_kernel, 2, 0.0), "greens": (L.sphere_greens_kernel, 3, 1.0),
                         "log": (L.planar_log_kernel, 4, 0.0), "delta3d": (L.delta3d_kernel, 5, 0.2),
                         "sphere_delta": (L.sphere_delta_kernel, 6, 0.2)}[name]
    kernel = make(1.0, param) if kind == 1 else make(param) if kind in (3, 5, 6) else make()
    src, tgt = _data(n_src, n_tgt, name in ("poisson", "log", "delta3d"))
    pick = np.unique(np.r_[:min(300, n_tgt), 0:n_tgt:37, n_tgt - 300:n_tgt])
    own = np.where(pick < n_src, pick, -1)
    got = _sum(ctx, kernel, L.LPM_PREC_F64, src, tgt, 3 if kind == 1 else 1, n_src)[:, pick]
    if n_src == 0:
        assert not got.any()
    elif kind == 1:
        assert rel_linf(got, oracle.bs_direct(src, tgt[pick], delta=param)) < 1e-12
    elif kind == 2:
        assert rel_linf(got[0], oracle.poisson_direct(src, tgt[pick])) < 1e-12
    else:
        ref = oracle.scalar_direct(kind, param, src, tgt[pick], own if kind in (3, 4) else None)
        assert rel_linf(got[0], ref) < 1e-12


@pytest.mark.parametrize("n_src,n_tgt", [(1, 148001), (256, 148001), (257, 147999), (257, 148001), (700, 300001),
                                         (1100, 300001), (2048, 148001), (2049, 148001)])
@pytest.mark.parametrize("scalar", [False, True])
def test_few_tiles_many_targets_f32(ctx, n_src, n_tgt, scalar):
    """Around the tiles and the targets per SM from which fewer groups share the tiles; the reference on the first, the
    last and every 37th target."""
    ctx.use_torch_stream()
    kernel = L.poisson_kernel() if scalar else L.biot_savart_kernel()
    src, tgt = _data(n_src, n_tgt, scalar)
    pick = np.unique(np.r_[:300, 0:n_tgt:37, n_tgt - 300:n_tgt])
    got = _sum(ctx, kernel, L.LPM_PREC_F32, src, tgt, 1 if scalar else 3, n_src)[:, pick]
    ref = oracle.poisson_direct(src, tgt[pick])[None] if scalar else oracle.bs_direct(src, tgt[pick])
    assert rel_l2(got, ref) < 5e-6
