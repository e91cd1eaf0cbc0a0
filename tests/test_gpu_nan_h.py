"""Particles and samples whose smoothing length is NaN.

A radius of NaN holds no pair: such a particle is no neighbour in the scatter
strategy, such a sample has none in the gather and symmetric ones (a particle's
NaN leaves the sample's radius to decide in the symmetric one).  The oracle's
neighbours, for both loops of the leaf tests, both precisions and element
types, and the single kernel's results.  The other particles share one h, and
samples of the symmetric strategy have no smaller one: a NaN below a node hides
the other h there from the node's scale, and no pair may hang on that.
"""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if not has_gpu():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import oracle as O  # noqa: E402
from partia_b200 import _lib as L  # noqa: E402
from partia_b200.engine import CatalogC, Context  # noqa: E402

PRECS = [L.PSB_PREC_FP64, L.PSB_PREC_FP32C]
STRATEGIES = [L.PSB_GATHER, L.PSB_SCATTER, L.PSB_SYMMETRIC]


def particles(n, seed, h, dtype, share=0.1):
    rng = np.random.default_rng(seed)
    x, y, z = rng.random((3, n))
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    hh = np.full(n, h)
    hh[rng.random(n) < share] = np.nan
    cols = [np.sin(3 * x) + y, rng.standard_normal(n)]
    return [a.astype(dtype) for a in (x, y, z, m, hh, rho)], [c.astype(dtype) for c in cols]


def pair(arrs, cols, dtype):
    orc = O.Oracle(*arrs, cols=cols, dtype=dtype)
    ctx = Context(0)
    ctx.set_particles(*arrs, cols=cols)
    ctx.build(want_perm=False)
    return orc, ctx


def check(orc, ctx, s, dtype, strategy, prec, hmode, hs=None):
    count, _, _ = orc.digest(s, strategy=strategy, hmode=hmode, hs=hs)
    cat = CatalogC(scalars=[0, 1], shepard=[0, 1], grads=[1])
    kw = dict(strategy=strategy, hmode=hmode, prec=prec, hs=hs)
    got = ctx.interp_points(*s, cat, **kw)
    assert ctx.last_stats.pairs == int(count.sum())
    dens = ctx.density(*s, **kw)
    assert not np.isnan(dens[count == 0]).any()
    ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
    one, done = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
    assert ctx.last_stats.pairs == int(count.sum())
    ctx.extra_flags = 0
    for a, b in zip([*got, dens], [*one, done]):
        if dtype == np.float64:
            assert np.array_equal(a, b, equal_nan=True)
        else:  # the parity tests' bound between the two for float inputs
            assert np.array_equal(np.isnan(a), np.isnan(b))
            f = ~np.isnan(b)
            assert not f.any() or np.abs(a[f] - b[f]).max() <= 1e-6 * np.abs(b[f]).max()


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("strategy", STRATEGIES)
@pytest.mark.parametrize("seed,root_nan", [(57, False), (50, True)])
def test_particles_without_a_radius(seed, root_nan, strategy, dtype, prec):
    """Close samples (a tile's samples against every leaf), loose and scattered
    ones (leaf by leaf, and node tests sample by sample); with a NaN for the
    largest h of the tree and without."""
    rng = np.random.default_rng(51)
    arrs, cols = particles(4000, seed, 0.08, dtype)
    orc, ctx = pair(arrs, cols, dtype)
    assert np.isnan(orc.tree()["node_scale"][0]) == root_nan
    close = tuple((0.35 + 0.3 * rng.random((3, 140_000))).astype(dtype))  # 32 samples a warp
    loose = tuple(rng.random((3, 700)).astype(dtype))
    far = tuple(rng.uniform(-1, 2, (3, 700)).astype(dtype))
    for s in (close, loose, far):
        check(orc, ctx, s, dtype, strategy, prec, L.PSB_H_CONSTANT, np.array([0.085], dtype=dtype))
        check(orc, ctx, s, dtype, strategy, prec, L.PSB_H_NEAREST)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("strategy", STRATEGIES)
def test_samples_without_a_radius(strategy, prec):
    rng = np.random.default_rng(52)
    arrs, cols = particles(4000, 53, 0.08, np.float64, share=0.0)
    orc, ctx = pair(arrs, cols, np.float64)
    s = tuple(rng.random((3, 3000)))
    hs = rng.uniform(0.05, 0.1, 3000)
    hs[::7] = np.nan
    check(orc, ctx, s, np.float64, strategy, prec, L.PSB_H_PER_SAMPLE, hs)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("strategy", [L.PSB_SCATTER, L.PSB_SYMMETRIC])
def test_edge_of_the_support_beside_them(strategy, sign, dtype, prec):
    """Samples on the support edge of particles whose span holds a NaN (or a
    negative h, whose square is the radius): the exact test decides there."""
    g = np.arange(12) * 0.1
    x, y, z = (a.ravel() for a in np.meshgrid(g, g, g, indexing="ij"))
    n = len(x)
    rng = np.random.default_rng(54)
    for k in (1, 2, 3):
        h = np.full(n, 0.05 * np.sqrt(k))
        if sign > 0:
            h[rng.random(n) < 0.2] = np.nan
        else:
            h[rng.random(n) < 0.2] *= -1
        arrs = [a.astype(dtype) for a in (x, y, z, np.full(n, 1.0 / n), h, np.ones(n))]
        orc, ctx = pair(arrs, [arrs[5]], dtype)
        s = tuple(np.concatenate([a[::3], a[1::7]]) for a in arrs[:3])
        hs = np.array([0.05 * np.sqrt(k)], dtype=dtype)
        count, _, _ = orc.digest(s, strategy=strategy, hmode=O.H_CONSTANT, hs=hs)
        ctx.interp_points(*s, CatalogC(scalars=[0], shepard=[0]), strategy=strategy, hmode=L.PSB_H_CONSTANT, hs=hs,
                          prec=prec)
        assert ctx.last_stats.pairs == int(count.sum()), k


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("nl", [300, 20_000])
@pytest.mark.parametrize("strategy", STRATEGIES)
def test_lines_without_a_radius(strategy, nl, prec):
    """Lines and particles with a NaN h: sight lines, and lines that run in tiles."""
    rng = np.random.default_rng(55)
    arrs, cols = particles(4000, 56, 0.08, np.float64)
    orc, ctx = pair(arrs, cols, np.float64)
    o = rng.uniform(0, 1, (3, nl))
    d = np.empty((3, nl))
    d[:] = [[0.0], [0.6], [0.8]]
    d[:, : nl // 4] = rng.standard_normal((3, nl // 4))
    d /= np.linalg.norm(d, axis=0)
    hs = rng.uniform(0.08, 0.1, nl)
    hs[::7] = np.nan
    count, _, _ = orc.digest(tuple(o), tuple(d), strategy=strategy, hmode=O.H_PER_SAMPLE, hs=hs)
    ctx.interp_lines(tuple(o), tuple(d), CatalogC(scalars=[0], shepard=[0]), strategy=strategy,
                     hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec)
    assert ctx.last_stats.pairs == int(count.sum())
    got, _, _ = ctx.digest(tuple(o), tuple(d), strategy=strategy, hmode=L.PSB_H_PER_SAMPLE, hs=hs,
                            fp32c=prec == L.PSB_PREC_FP32C)
    assert np.array_equal(got, count)
