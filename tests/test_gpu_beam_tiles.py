"""Beams over strongly clumped particles: tiles by eight lanes a line (512 to
1535 tiles) or one (more), those through the clumps handed to a warp per line on
a stream of its own.  Every line has the bits of the same line in a call that
takes a warp for each, and the pairs are the oracle's.
"""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if not has_gpu():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import oracle as O  # noqa: E402
from partia_b200 import _lib as L  # noqa: E402
from partia_b200 import workloads as W  # noqa: E402
from partia_b200.engine import CatalogC, Context  # noqa: E402


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("strategy", [L.PSB_GATHER, L.PSB_SCATTER, L.PSB_SYMMETRIC])
@pytest.mark.parametrize("nx,ny", [(251, 125), (531, 261)])  # 1024 and 4422 tiles of 8 x 4 lines
def test_heavy_tiles_beside_the_others(nx, ny, strategy, prec):
    rng = np.random.default_rng(91)
    n = 30_000
    cen = rng.uniform(0.2, 0.8, (4, 3))
    p = cen[rng.integers(0, 4, n)] + 0.004 * rng.standard_normal((n, 3))
    p[: n // 5] = rng.random((n // 5, 3))
    h = np.full(n, 0.0008)
    h[: n // 5] = 0.04
    m, rho = np.full(n, 1.0 / n), rng.uniform(0.5, 2.0, n)
    cols = [rng.standard_normal(n) for _ in range(2)]
    arrs = [np.ascontiguousarray(p[:, k]) for k in range(3)] + [m, h, rho]
    ctx = Context(0)
    ctx.set_particles(*arrs, cols=cols)
    ctx.build(want_perm=False)
    fr = W.Frame((0.5, 0.5, 0.5), (0.3, -0.2, 1.0), (1.0, 0.0, -0.3))
    fr.rotate(0.2, 0.1, -0.4)
    farr = fr.as_array()
    prm = np.array([-0.4, 0.45, -0.45, 0.4])
    cat = CatalogC(scalars=[0, 1], shepard=[0, 1])
    kw = dict(strategy=strategy, hmode=L.PSB_H_CONSTANT, hs=np.array([0.006]), prec=prec)
    # the tile with the most particles has many times the mean (1.5 to 3 times the cost is handed over)
    v = p - farr[:3]
    i = (v @ farr[3:6] - prm[0]) / (prm[1] - prm[0]) * (nx - 1) // 8
    j = (v @ farr[6:9] - prm[2]) / (prm[3] - prm[2]) * (ny - 1) // 4
    nbx, nby = (nx + 7) // 8, (ny + 3) // 4
    on = (i >= 0) & (i < nbx) & (j >= 0) & (j < nby)
    per_tile = np.bincount((i + nbx * j)[on].astype(np.int64), minlength=nbx * nby)
    assert per_tile.max() > 20 * per_tile.mean()
    got = ctx.interp_beam(farr, prm, nx, ny, cat, **kw)
    pairs = ctx.last_stats.pairs
    ox = W.plane_coordinates(farr, (prm[0], prm[1], nx), (prm[2], prm[3], ny))
    fw = tuple(np.full(nx * ny, farr[9 + c]) for c in range(3))
    count, _, _ = O.Oracle(*arrs, cols=cols).digest(ox, fw, strategy=strategy, hmode=O.H_CONSTANT, hs=kw["hs"])
    assert pairs == int(count.sum())
    for a in range(0, nx * ny, 16_000):  # 500 tiles: a warp per line
        at = slice(a, a + 16_000)
        one = ctx.interp_lines(tuple(v[at] for v in ox), tuple(v[at] for v in fw), cat, **kw)
        for k in range(2):
            assert np.array_equal(one[k], got[k][at], equal_nan=True), (a, k)
