"""The point path's walk, list parts and large-neighbourhood samples.

 * Samples whose accepted spans fill one list part, several, and more than the
   tile's walk keeps (k_heavy), mixed in one tile: against the oracle, and bit
   for bit against the single kernel, which sums in the same parts.
 * Sample sets that a warp's box fits badly (scattered samples, a tile of
   which one is far away), calls of a few samples (fewer samples per warp) and
   trees of a few particles.
 * Samples that the float tests do not cover (NaN, infinite and huge
   coordinates and h) and particle sets outside their range.
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

FP64_TOL = 1e-12  # the parity tests' bound
SPEC = dict(scalars=[0, 1], shepard=[0, 1], grads=[-1, 1], divs=[1, 2, 3], curls=[1, 2, 3])


def rel_err(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    assert np.array_equal(np.isnan(a), np.isnan(b)), "NaN masks differ"
    f = ~np.isnan(b)
    return float(np.max(np.abs(a[f] - b[f])) / max(np.max(np.abs(b[f])), 1e-300)) if f.any() else 0.0


def particles(n, seed, dtype=np.float64):
    rng = np.random.default_rng(seed)
    x, y, z = rng.random(n), rng.random(n), rng.random(n)
    m = rng.uniform(0.5, 1.5, n) / n
    h = 1.2 * (1.0 / n) ** (1 / 3) * rng.uniform(0.5, 2.0, n)
    rho = rng.uniform(0.5, 2.0, n)
    cols = [rho.copy(), np.sin(3 * x) + y, -y + 0.1 * rng.standard_normal(n), x + 0.1 * rng.standard_normal(n)]
    return [a.astype(dtype) for a in (x, y, z, m, h, rho)], [c.astype(dtype) for c in cols]


def context(arrs, cols, kernel=L.PSB_KERNEL_M4):
    ctx = Context(0)
    ctx.set_particles(*arrs, cols=cols, kernel=kernel)
    ctx.build(want_perm=False)
    return ctx


@pytest.mark.parametrize("strategy", [L.PSB_GATHER, L.PSB_SYMMETRIC])
@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("kid", [L.PSB_KERNEL_M4, L.PSB_KERNEL_M6])
@pytest.mark.parametrize("ns", [70, 5000])
def test_list_parts_and_heavy_samples(ns, kid, prec, strategy):
    """h up to 0.3 of the box: one to about 900 accepted spans a sample."""
    arrs, cols = particles(20_000, 5)
    rng = np.random.default_rng(6)
    s = tuple(rng.random(ns) for _ in range(3))
    hs = rng.choice([0.01, 0.03, 0.06, 0.12, 0.3], ns, p=[0.5, 0.3, 0.1, 0.09, 0.01])
    hs[:2] = 0.3, 0.12
    orc = O.Oracle(*arrs, cols=cols, kernel=kid)
    ref = orc.interp_points(*s, O.Catalog(**SPEC), strategy=strategy, hmode=O.H_PER_SAMPLE, hs=hs)
    count, _, _ = orc.digest(s, strategy=strategy, hmode=O.H_PER_SAMPLE, hs=hs)
    ctx = context(arrs, cols, kid)
    cat = CatalogC(**SPEC)
    kw = dict(strategy=strategy, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec)
    got = ctx.interp_points(*s, cat, **kw)
    assert ctx.last_stats.pairs == int(count.sum())
    dens = ctx.density(*s, **kw)
    ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
    one = ctx.interp_points(*s, cat, **kw)
    done = ctx.density(*s, **kw)
    for k in range(cat.L):
        if prec == L.PSB_PREC_FP64:
            assert rel_err(got[k], ref[k]) <= FP64_TOL, k
        assert np.array_equal(got[k], one[k], equal_nan=True), k
    assert np.array_equal(dens, done)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("kid", [L.PSB_KERNEL_M4, L.PSB_KERNEL_M5])
def test_small_calls_have_the_bits_of_large_ones(kid, prec, dtype):
    """Up to 4096 samples a warp sums each sample, above that a lane: the same
    pairs, rounded alike and added in the same order, with the same parts."""
    arrs, cols = particles(20_000, 11, dtype)
    rng = np.random.default_rng(12)
    ns = 4097
    s = tuple(rng.random(ns).astype(dtype) for _ in range(3))
    hs = rng.choice([0.01, 0.03, 0.06, 0.12, 0.3], ns, p=[0.5, 0.3, 0.15, 0.04, 0.01]).astype(dtype)
    ctx = context(arrs, cols, kid)
    cat = CatalogC(**SPEC)
    for strategy in (L.PSB_GATHER, L.PSB_SCATTER, L.PSB_SYMMETRIC):
        kw = dict(strategy=strategy, hmode=L.PSB_H_PER_SAMPLE, prec=prec)
        large = ctx.interp_points(*s, cat, hs=hs, **kw) + [ctx.density(*s, hs=hs, **kw)]
        for k0, k1 in ((0, 4096), (4094, 4097)):
            t = tuple(a[k0:k1] for a in s)
            small = ctx.interp_points(*t, cat, hs=hs[k0:k1], **kw) + [ctx.density(*t, hs=hs[k0:k1], **kw)]
            for k, (a, b) in enumerate(zip(small, large)):
                assert np.array_equal(a, b[k0:k1], equal_nan=True), (strategy, k)


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
def test_heavy_samples_of_float_particles(prec):
    """Float particles: equal to the single kernel to a float rounding, whose parts these are."""
    arrs, cols = particles(20_000, 7, np.float32)
    rng = np.random.default_rng(8)
    s = tuple(rng.random(300).astype(np.float32) for _ in range(3))
    hs = rng.choice([0.01, 0.06, 0.3], 300).astype(np.float32)
    ctx = context(arrs, cols)
    cat = CatalogC(**SPEC)
    kw = dict(strategy=L.PSB_SYMMETRIC, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec)
    got = ctx.interp_points(*s, cat, **kw)
    pairs = ctx.last_stats.pairs
    ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
    one = ctx.interp_points(*s, cat, **kw)
    assert ctx.last_stats.pairs == pairs
    for k in range(cat.L):
        assert rel_err(got[k], one[k]) <= 1e-6, k


@pytest.mark.parametrize("n", [1, 2, 32, 33, 65, 4000])
@pytest.mark.parametrize("ns", [1, 31, 33, 200])
def test_few_samples_and_scattered_samples(n, ns):
    """Samples over ten times the box, so that no box fits a warp's samples: the
    oracle's neighbours, and the single kernel's bits (a field of one or two
    neighbours is a difference of equal terms, so a relative bound says nothing)."""
    arrs, cols = particles(n, 9)
    rng = np.random.default_rng(10 + ns)
    s = tuple(rng.uniform(-5, 6, ns) if ns > 1 else rng.random(ns) for _ in range(3))
    orc = O.Oracle(*arrs, cols=cols)
    ctx = context(arrs, cols)
    cat = CatalogC(**SPEC)
    for strategy in (L.PSB_GATHER, L.PSB_SCATTER, L.PSB_SYMMETRIC):
        count, _, _ = orc.digest(s, strategy=strategy, hmode=O.H_NEAREST)
        for prec in (L.PSB_PREC_FP64, L.PSB_PREC_FP32C):
            kw = dict(strategy=strategy, hmode=L.PSB_H_NEAREST, prec=prec)
            got = ctx.interp_points(*s, cat, **kw)
            assert ctx.last_stats.pairs == int(count.sum())
            ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
            one = ctx.interp_points(*s, cat, **kw)
            ctx.extra_flags = 0
            for k in range(cat.L):
                assert np.array_equal(got[k], one[k], equal_nan=True), (strategy, prec, k)


def test_samples_outside_the_float_tests():
    """NaN, infinite and huge positions and h leave the other samples' results as they are."""
    arrs, cols = particles(5000, 11)
    rng = np.random.default_rng(12)
    ns = 400
    s = [rng.random(ns) for _ in range(3)]
    hs = rng.uniform(0.02, 0.06, ns)
    ctx = context(arrs, cols)
    cat = CatalogC(**SPEC)
    clean = ctx.interp_points(*s, cat, strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs)
    bad = {3: np.nan, 40: np.inf, 77: -np.inf, 130: 1e300, 200: -1e25}
    for i, v in bad.items():
        s[i % 3][i] = v
    hb = hs.copy()
    hb[[250, 300]] = np.nan, -0.03
    got = ctx.interp_points(*s, cat, strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hb)
    for k in range(cat.L):
        assert np.all(np.isnan(got[k][[*bad, 250]])), k
    same = np.setdiff1d(np.arange(ns), [*bad, 250, 300])
    for k in range(cat.L):
        assert rel_err(got[k][same], clean[k][same]) <= 1e-14, k


@pytest.mark.parametrize("scale", [1e-15, 1e-9, 1e12, 1e17])
def test_particle_sets_of_any_scale(scale):
    """The kernel sums scale with the lengths: rho (plain sum of A m/rho W) is
    scale free, inside and outside the float tests' range."""
    arrs, cols = particles(3000, 13)
    rng = np.random.default_rng(14)
    s = [rng.random(300) for _ in range(3)]
    spec = dict(scalars=[1], shepard=[1])
    ref = context(arrs, cols).interp_points(*s, CatalogC(**spec), strategy=L.PSB_SYMMETRIC)
    big = [a * scale for a in arrs[:3]] + [arrs[3], arrs[4] * scale, arrs[5]]
    got = context(big, cols).interp_points(*[a * scale for a in s], CatalogC(**spec), strategy=L.PSB_SYMMETRIC)
    # a Shepard mean of 64-bit coordinates rounded at another scale: 1e-16 of
    # the separations, amplified at the support edge by less than 1e3
    assert rel_err(got[0], ref[0]) <= 1e-12


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("nl", [1, 33, 1000, 40_000])
def test_lines_alone_and_in_tiles(nl, prec):
    """Sight lines in every direction and a bundle of parallel ones, below and
    above the size from which a tile's lines may run together; seven columns.  Each line's bits are the same alone (a
    call of one) and among the others."""
    arrs, cols = particles(20_000, 15)
    rng = np.random.default_rng(16)
    cols = cols + [rng.random(20_000) for _ in range(3)]
    o = rng.uniform(-0.2, 1.2, (3, nl))
    d = rng.standard_normal((3, nl))
    d /= np.linalg.norm(d, axis=0)
    d[:, nl // 4:nl // 2] = [[0.0], [0.6], [0.8]]
    o[:, nl // 4:nl // 2] *= 0.1  # close to one another
    spec = dict(scalars=list(range(7)), shepard=[0, 1, 1, 1, 0, 1, 0])
    orc = O.Oracle(*arrs, cols=cols)
    ctx = context(arrs, cols)
    cat = CatalogC(**spec)
    got = ctx.interp_lines(tuple(o), tuple(d), cat, prec=prec)
    pairs = ctx.last_stats.pairs
    m = min(nl, 2000)
    at = rng.choice(nl, m, replace=False)
    ref = orc.interp_lines(tuple(o[:, at]), tuple(d[:, at]), scalars=spec["scalars"], shepard=spec["shepard"],
                           strategy=O.SCATTER, hmode=O.H_PER_SAMPLE, hs=None)
    tol = FP64_TOL if prec == L.PSB_PREC_FP64 else 4e-6  # the parity tests' bounds
    if nl > 1:
        for k in range(cat.L):
            assert rel_err(got[k][at], ref[k]) <= tol, k
    if nl <= 1000:
        count, _, _ = orc.digest(tuple(o), tuple(d), strategy=O.SCATTER, hmode=O.H_PER_SAMPLE)
        assert pairs == int(count.sum())
    for i in at[:20]:
        one = ctx.interp_lines(tuple(o[:, i:i + 1]), tuple(d[:, i:i + 1]), cat, prec=prec)
        for k in range(cat.L):
            assert np.array_equal(one[k], got[k][i:i + 1], equal_nan=True), (i, k)


def test_lines_that_are_not_unit_vectors():
    """The formula D^2 - (D.m)^2 holds for any m: the reference's pairs, in FP64."""
    arrs, cols = particles(5000, 17)
    rng = np.random.default_rng(18)
    o, d = rng.random((3, 50)), rng.standard_normal((3, 50))
    d *= rng.uniform(0.9, 0.999, 50) / np.linalg.norm(d, axis=0)
    orc = O.Oracle(*arrs, cols=cols)
    ctx = context(arrs, cols)
    got = ctx.interp_lines(tuple(o), tuple(d), CatalogC(scalars=[0, 1], shepard=[0, 1]))
    count, _, _ = orc.digest(tuple(o), tuple(d), strategy=O.SCATTER, hmode=O.H_PER_SAMPLE)
    ref = orc.interp_lines(tuple(o), tuple(d), scalars=[0, 1], shepard=[0, 1], strategy=O.SCATTER,
                           hmode=O.H_PER_SAMPLE, hs=None)
    assert ctx.last_stats.pairs == int(count.sum())
    for k in range(2):
        assert rel_err(got[k], ref[k]) <= FP64_TOL, k


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kc", [3, 5, 6, 7])
def test_column_counts(kc, dtype):
    """Every column count that has pair sums of its own: equal to the single kernel's."""
    arrs, cols = particles(3000, 19, dtype)
    rng = np.random.default_rng(20)
    cols = [rng.standard_normal(3000).astype(dtype) for _ in range(kc)]
    s = tuple(rng.random(500).astype(dtype) for _ in range(3))
    ctx = context(arrs, cols)
    cat = CatalogC(scalars=list(range(kc)), shepard=[k % 2 for k in range(kc)], grads=[-1, kc - 1])
    for prec in (L.PSB_PREC_FP64, L.PSB_PREC_FP32C):
        got = ctx.interp_points(*s, cat, strategy=L.PSB_SYMMETRIC, prec=prec)
        ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
        one = ctx.interp_points(*s, cat, strategy=L.PSB_SYMMETRIC, prec=prec)
        ctx.extra_flags = 0
        for k in range(cat.L):
            if dtype == np.float64:
                assert np.array_equal(got[k], one[k], equal_nan=True), (prec, k)
            else:  # (the parity tests' bound between the two for float inputs)
                assert rel_err(got[k], one[k]) <= 1e-6, (prec, k)


def test_float_decisions_on_the_support_edge():
    """Float particles on a lattice with radii that are its distances: the sum
    of squares rounds at every step, and a fused one decides otherwise."""
    g = np.arange(12, dtype=np.float32) * np.float32(0.1)
    x, y, z = (a.ravel().astype(np.float32) for a in np.meshgrid(g, g, g, indexing="ij"))
    n = len(x)
    one = np.ones(n, dtype=np.float32)
    rng = np.random.default_rng(21)
    h = (np.float32(0.05) * np.sqrt(rng.integers(1, 9, n))).astype(np.float32)
    ctx = context([x, y, z, one / n, h, one], [one])
    s = tuple(np.concatenate([a[::3], a[1::7]]) for a in (x, y, z))
    orc = O.Oracle(x, y, z, one / n, h, one, cols=[one], dtype=np.float32)
    for strategy in (L.PSB_GATHER, L.PSB_SCATTER, L.PSB_SYMMETRIC):
        for hs in ([0.05], [0.0707106781], [0.1], [0.111803398]):
            kw = dict(strategy=strategy, hmode=L.PSB_H_CONSTANT, hs=np.array(hs, dtype=np.float32))
            ctx.interp_points(*s, CatalogC(scalars=[0], shepard=[0]), **kw)
            count, _, _ = orc.digest(s, **kw)
            assert ctx.last_stats.pairs == int(count.sum()), (strategy, hs)


@pytest.mark.parametrize("ns", [500, 4000, 9000])
def test_out_of_range_samples_leave_their_neighbours_lists(ns):
    """Samples outside the float range in every tile and in small calls' warps of
    a few samples: the single kernel takes them, once each (pairs are counted
    once), and the others keep their results."""
    arrs, cols = particles(20_000, 13)
    rng = np.random.default_rng(14)
    s = [rng.random(ns) for _ in range(3)]
    s[1][rng.random(ns) < 0.2] = 1e19
    hs = np.full(ns, 0.05)
    ctx = context(arrs, cols)
    cat = CatalogC(**SPEC)
    for prec in (L.PSB_PREC_FP64, L.PSB_PREC_FP32C):
        kw = dict(strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec)
        ctx.extra_flags = 0
        got = ctx.interp_points(*s, cat, **kw)
        pairs = ctx.last_stats.pairs
        ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
        one = ctx.interp_points(*s, cat, **kw)
        assert ctx.last_stats.pairs == pairs
        for k in range(cat.L):
            assert np.array_equal(got[k], one[k], equal_nan=True), (prec, k)


def test_more_large_neighbourhoods_than_the_pool_holds():
    """20,000 samples that each reach most of 30,000 particles: more entries than
    the lists hold, so the single kernel sums the rest; every pair counted once."""
    arrs, cols = particles(30_000, 15)
    rng = np.random.default_rng(16)
    s = [rng.random(20_000) for _ in range(3)]
    hs = np.full(20_000, 0.3)
    hs[rng.random(20_000) < 0.3] = 0.02
    ctx = context(arrs, cols)
    kw = dict(strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=L.PSB_PREC_FP32C)
    cat = CatalogC(scalars=[0, 1], grads=[-1, 1])
    got, dens = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
    pairs = ctx.last_stats.pairs
    ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
    one, done = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
    assert ctx.last_stats.pairs == pairs
    for k in range(cat.L):
        assert np.array_equal(got[k], one[k], equal_nan=True), k
    assert np.array_equal(dens, done)
