"""Many samples of large neighbourhoods: k_heavy's blocks take several in turn,
of different sizes, so that a block's threads that run ahead meet the next
sample while others still place the last one's entries.  Bit for bit against
the single kernel, and the oracle's pair counts.
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


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("kid", [L.PSB_KERNEL_M4, L.PSB_KERNEL_M6])
def test_blocks_take_several_heavy_samples_in_turn(kid, prec):
    rng = np.random.default_rng(41)
    n, ns = 20_000, 1500  # five samples to each of k_heavy's blocks
    x, y, z = rng.random((3, n))
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    h = 1.2 * n ** (-1 / 3) * rng.uniform(0.5, 2.0, n)
    cols = [rng.standard_normal(n) for _ in range(2)]
    s = tuple(rng.random((3, ns)))
    hs = rng.uniform(0.1, 0.18, ns) * (2.0 if kid == L.PSB_KERNEL_M4 else 1.4)
    count, _, _ = O.Oracle(x, y, z, m, h, rho, cols=cols, kernel=kid).digest(
        s, strategy=O.GATHER, hmode=O.H_PER_SAMPLE, hs=hs)
    ctx = Context(0)
    ctx.set_particles(x, y, z, m, h, rho, cols, kernel=kid)
    ctx.build(want_perm=False)
    cat = CatalogC(scalars=[0, 1], shepard=[0, 1], grads=[-1, 1])
    kw = dict(strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec)
    ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
    one, done = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
    ctx.extra_flags = 0
    for _ in range(5):
        got, dens = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
        assert ctx.last_stats.pairs == int(count.sum())
        for k in range(cat.L):
            assert np.array_equal(got[k], one[k], equal_nan=True), k
        assert np.array_equal(dens, done)


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("kid", [L.PSB_KERNEL_M4, L.PSB_KERNEL_M5, L.PSB_KERNEL_C4])
@pytest.mark.parametrize("ns", [40, 6000])
@pytest.mark.parametrize("kc", [1, 8])
def test_pair_sums_by_a_warp(kc, ns, kid, prec):
    """Parts of 1 to 1024 pairs, in windows of 32 pairs whatever entries they
    come from; up to 40 sums, two to a lane.  Small calls (a warp sums each
    sample) and the samples of several parts in larger FP32C ones."""
    rng = np.random.default_rng(43)
    n = 8000
    x, y, z = rng.random((3, n))
    x[:500] = 0.5 + 1e-3 * rng.random(500)  # full spans
    y[:500] = 0.5 + 1e-3 * rng.random(500)
    z[:500] = 0.5 + 1e-3 * rng.random(500)
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    h = 1.2 * n ** (-1 / 3) * rng.uniform(0.5, 2.0, n)
    cols = [rng.standard_normal(n) for _ in range(kc)]
    s = rng.random((3, ns))
    s[:, ::5] = 0.5 + 1e-2 * rng.standard_normal((3, len(s[0, ::5])))
    hs = rng.choice([0.005, 0.02, 0.05, 0.1, 0.2], ns)
    ctx = Context(0)
    ctx.set_particles(x, y, z, m, h, rho, cols, kernel=kid)
    ctx.build(want_perm=False)
    cat = CatalogC(scalars=range(kc), shepard=[0] * kc, grads=[-1, *range(kc)])
    for strategy in (L.PSB_GATHER, L.PSB_SCATTER, L.PSB_SYMMETRIC):
        kw = dict(strategy=strategy, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec)
        got, dens = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
        ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
        one, done = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
        ctx.extra_flags = 0
        for k in range(cat.L):
            assert np.array_equal(got[k], one[k], equal_nan=True), (strategy, k)
        assert np.array_equal(dens, done)


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("ns", [50, 6000])
@pytest.mark.parametrize("reach", [0.03, 0.3])
def test_statistics_count_all_forms(reach, ns, prec):
    """A loop iteration of a warp holds at most 32 pairs, a span test at most 32
    leaves, whichever kernel takes the sample."""
    rng = np.random.default_rng(45)
    n = 20_000
    x, y, z = rng.random((3, n))
    one = np.ones(n)
    ctx = Context(0)
    ctx.set_particles(x, y, z, one / n, np.full(n, 0.05), one, [one])
    ctx.build(want_perm=False)
    s = tuple(rng.random((3, ns)))
    hs = np.full(ns, 0.03)
    hs[::10] = reach
    kw = dict(strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec)
    for call in (lambda: ctx.interp_points(*s, CatalogC(scalars=[0], shepard=[0]), **kw), lambda: ctx.density(*s, **kw)):
        call()
        st = ctx.last_stats
        assert 0 < st.pairs <= 32 * st.body_iters
        assert st.pairs <= 32 * st.span_tests and st.spans <= st.span_tests


@pytest.mark.parametrize("kid", [L.PSB_KERNEL_M4, L.PSB_KERNEL_M6])
@pytest.mark.parametrize("kc", [1, 3, 6])
def test_many_samples_of_a_few_parts(kc, kid):
    """More samples of several parts in a batch than go to a lane each in FP32C,
    most of them of two to four parts and some of more: the single kernel's bits."""
    rng = np.random.default_rng(47)
    n, ns = 4000, 300_000  # four batches of 75,000
    x, y, z = rng.random((3, n))
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    h = 1.2 * n ** (-1 / 3) * rng.uniform(0.5, 2.0, n)
    cols = [rng.standard_normal(n) for _ in range(kc)]
    s = rng.random((3, ns))
    hs = rng.choice([0.12, 0.16, 0.3], ns, p=[0.5, 0.45, 0.05])
    ctx = Context(0)
    ctx.set_particles(x, y, z, m, h, rho, cols, kernel=kid)
    ctx.build(want_perm=False)
    cat = CatalogC(scalars=range(kc), shepard=[0] * kc, grads=[-1, kc - 1])
    kw = dict(strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=L.PSB_PREC_FP32C)
    ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
    one, done = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
    pairs = ctx.last_stats.pairs
    ctx.extra_flags = 0
    for _ in range(3):  # (the pool grows to the need)
        got, dens = ctx.interp_points(*s, cat, **kw), ctx.density(*s, **kw)
        assert ctx.last_stats.pairs == pairs
        for a, b in zip([*got, dens], [*one, done]):
            assert np.array_equal(a, b, equal_nan=True)
