"""Sight lines that each meet much of a small set: tiles take them together
whatever their directions, from some share of the spans and some number of tiles
on; lines that are no unit vectors keep a warp of their own.  Every
line has the bits of the same line in a call of few lines, which takes a warp
for each, and the pairs are the oracle's.
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
@pytest.mark.parametrize("strategy", [L.PSB_GATHER, L.PSB_SCATTER, L.PSB_SYMMETRIC])
@pytest.mark.parametrize("n,nl", [(1, 20_000), (300, 40_000), (1500, 50_003), (1500, 140_000)])
def test_lines_in_any_direction_through_a_small_set(n, nl, strategy, prec):
    rng = np.random.default_rng(101)
    x, y, z = rng.random((3, n))
    m, rho = np.full(n, 1.0 / n), rng.uniform(0.5, 2.0, n)
    h = 1.2 * n ** (-1 / 3) * rng.uniform(0.3, 1.5, n)
    cols = [rng.standard_normal(n) for _ in range(2)]
    ctx = Context(0)
    ctx.set_particles(x, y, z, m, h, rho, cols)
    ctx.build(want_perm=False)
    o = rng.uniform(-0.1, 1.1, (3, nl))
    d = rng.standard_normal((3, nl))
    d /= np.linalg.norm(d, axis=0)
    d[:, ::1001] *= 0.97  # not a unit vector
    hs = rng.uniform(0.02, 0.2, nl)
    cat = CatalogC(scalars=[0, 1], shepard=[0, 1])
    kw = dict(strategy=strategy, hmode=L.PSB_H_PER_SAMPLE, prec=prec)
    got = ctx.interp_lines(tuple(o), tuple(d), cat, hs=hs, **kw)
    pairs = ctx.last_stats.pairs
    count, _, _ = O.Oracle(x, y, z, m, h, rho, cols=cols).digest(
        tuple(o), tuple(d), strategy=strategy, hmode=O.H_PER_SAMPLE, hs=hs)
    assert pairs == int(count.sum())
    if nl == 140_000:  # together: some pairs are undecided in float (a warp per line decides all in double)
        assert ctx.last_stats.exact_retests > 0
    for a in range(0, nl, 9000):  # 282 tiles: a warp per line
        at = slice(a, min(a + 9000, nl))
        one = ctx.interp_lines(tuple(o[:, at]), tuple(d[:, at]), cat, hs=hs[at], **kw)
        assert ctx.last_stats.exact_retests == 0
        for k in range(2):
            assert np.array_equal(one[k], got[k][at], equal_nan=True), (a, k)
