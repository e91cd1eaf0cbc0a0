"""Particle sets in any unit of length, and sets of no extent.

Outside the range of the float tests (coordinates and h above 1e18, an extent
below 1e-12: a galaxy in centimetres, an atom in metres) the lists' walk tests
in the particles' own arithmetic.  The oracle's neighbours, the single kernel's
bits, and the same passes as for the set at unit scale.
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

STRATEGIES = [L.PSB_GATHER, L.PSB_SCATTER, L.PSB_SYMMETRIC]
SPEC = dict(scalars=[0, 1], shepard=[0, 1], grads=[-1, 1])


def particles(n, seed, scale, dtype):
    rng = np.random.default_rng(seed)
    x, y, z = rng.random((3, n)) * scale
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    h = 1.2 * n ** (-1 / 3) * rng.uniform(0.5, 2.0, n) * scale
    return [a.astype(dtype) for a in (x, y, z, m, h, rho)], [rng.standard_normal(n).astype(dtype) for _ in range(2)]


def context(arrs, cols, kernel=L.PSB_KERNEL_M4):
    ctx = Context(0)
    ctx.set_particles(*arrs, cols=cols, kernel=kernel)
    ctx.build(want_perm=False)
    return ctx


def same(a, b, dtype):
    if dtype == np.float64:
        return np.array_equal(a, b, equal_nan=True)
    f = np.isfinite(b)  # float inputs: the parity tests' bound between the two
    return np.array_equal(f, np.isfinite(a)) and (not f.any() or np.abs(a[f] - b[f]).max() <= 1e-6 * np.abs(b[f]).max())


@pytest.mark.parametrize("ns", [300, 20_000])
@pytest.mark.parametrize("dtype,prec,scale", [
    *[(np.float64, L.PSB_PREC_FP64, s) for s in (1e-120, 1e-40, 1e-14, 2e15, 0.9e18, 1e22, 1e120)],
    *[(np.float64, L.PSB_PREC_FP32C, s) for s in (1e-14, 2e15, 0.9e18, 1e22)],
    *[(np.float32, p, s) for p in (L.PSB_PREC_FP64, L.PSB_PREC_FP32C) for s in (1e-14, 2e15, 0.9e18, 1e19)]])
def test_sets_outside_the_float_tests_take_the_lists(dtype, prec, scale, ns):
    arrs, cols = particles(4000, 71, scale, dtype)
    rng = np.random.default_rng(72)
    s = tuple((rng.uniform(-0.1, 1.1, (3, ns)) * scale).astype(dtype))  # (0.9e18: up to the samples' limit)
    hs = (rng.choice([0.02, 0.06, 0.12, 0.3], ns, p=[0.6, 0.3, 0.09, 0.01]) * scale).astype(dtype)
    orc = O.Oracle(*arrs, cols=cols, dtype=dtype)
    ctx = context(arrs, cols)
    unit = context(*particles(4000, 71, 1.0, dtype))
    cat = CatalogC(**SPEC)
    for strategy in STRATEGIES:
        for kw in (dict(hmode=L.PSB_H_NEAREST), dict(hmode=L.PSB_H_PER_SAMPLE, hs=hs)):
            count, _, _ = orc.digest(s, strategy=strategy, **kw)
            kw = dict(kw, strategy=strategy, prec=prec)
            got, pairs, launches = ctx.interp_points(*s, cat, **kw), ctx.last_stats.pairs, ctx.last_stats.launches
            dens = ctx.density(*s, **kw)
            assert pairs == int(count.sum()) and ctx.last_stats.pairs == pairs
            unit.interp_points(*s, cat, **kw)
            assert launches == unit.last_stats.launches
            ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
            one, done = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
            ctx.extra_flags = 0
            for a, b in zip([*got, dens], [*one, done]):
                assert same(a, b, dtype), (strategy, kw["hmode"])


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [1, 2, 40, 3000])
def test_particles_in_one_place(n, dtype, prec):
    """No extent: one particle, and many at the same point."""
    rng = np.random.default_rng(73)
    arrs, cols = particles(n, 74, 1.0, dtype)
    for a in arrs[:3]:
        a[:] = 0.5
    s = rng.uniform(0, 1, (3, 200)).astype(dtype)
    s[:, :50] = 0.5 + 0.01 * rng.standard_normal((3, 50))
    s[:, :5] = 0.5
    s = tuple(s)
    orc = O.Oracle(*arrs, cols=cols, dtype=dtype)
    ctx = context(arrs, cols)
    cat = CatalogC(**SPEC)
    for strategy in STRATEGIES:
        count, _, _ = orc.digest(s, strategy=strategy, hmode=O.H_NEAREST)
        kw = dict(strategy=strategy, hmode=L.PSB_H_NEAREST, prec=prec)
        got, dens = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
        assert ctx.last_stats.pairs == int(count.sum())
        ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
        one, done = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
        ctx.extra_flags = 0
        for a, b in zip([*got, dens], [*one, done]):
            assert same(a, b, dtype), strategy


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("shift", [1e5, 3e6, 1e9])
def test_sets_far_from_the_origin(shift, prec):
    """A float's step at the coordinates from a fraction of the particles' spacing to
    far above the set's extent: the oracle's pairs, in about as many span tests as
    at the origin (where the float tests leave nothing out, every span is tested)."""
    n, ns = 4000, 3000
    arrs, cols = particles(n, 75, 1.0, np.float64)
    s = np.random.default_rng(76).random((3, ns))
    cat = CatalogC(**SPEC)
    near = context(arrs, cols)
    moved = [a + shift for a in arrs[:3]] + arrs[3:]
    orc, ctx = O.Oracle(*moved, cols=cols), context(moved, cols)
    for strategy in STRATEGIES:
        kw = dict(strategy=strategy, prec=prec)
        near.interp_points(*s, cat, **kw)
        ctx.interp_points(*(s + shift), cat, **kw)
        count, _, _ = orc.digest(tuple(s + shift), strategy=strategy)
        assert ctx.last_stats.pairs == int(count.sum())
        assert ctx.last_stats.span_tests <= 1.5 * near.last_stats.span_tests
