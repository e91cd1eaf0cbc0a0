"""The adjoint's pair sums in equal runs: a list block's pairs are dealt out to
the lanes whatever particles they belong to.  Blocks of fewer pairs than lanes,
of one particle with most of the pairs, and ordinary ones; catalogs of scalars,
of gradients, and with the density gradient; one to eight columns.  Against
the single kernel, which sums each particle in one lane (1e-12 of each
gradient's maximum, the adjoint tests' bound between the two), and against
the oracle (1e-10, the adjoint tests' bound).
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

CATS = {
    "scalar1": dict(scalars=[1], shepard=[1]),
    "scalar2": dict(scalars=[0, 2], shepard=[0, 1]),
    "gradient1": dict(grads=[1]),
    "gradient4": dict(scalars=[0], shepard=[0], grads=[0], divs=[1, 2, 3], curls=[1, 2, 3]),
    "full4": dict(scalars=[0], shepard=[1], grads=[-1, 2], divs=[1, 2, 3], curls=[1, 2, 3]),
    "full8": dict(scalars=list(range(8)), shepard=[0, 1] * 4, grads=[-1, 7], curls=[4, 5, 6]),
}


@pytest.mark.parametrize("cat", list(CATS))
@pytest.mark.parametrize("n,ns", [(40, 1), (3000, 5), (3000, 700), (33, 900)])
@pytest.mark.parametrize("strategy", [L.PSB_GATHER, L.PSB_SYMMETRIC])
def test_runs_match_one_lane_per_particle(cat, n, ns, strategy):
    rng = np.random.default_rng(n + ns)
    x, y, z = rng.random(n), rng.random(n), rng.random(n)
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    h = 1.2 * n ** (-1 / 3) * rng.uniform(0.5, 1.5, n)
    h[:: max(1, n // 3)] *= 4  # a few particles with most of the pairs
    cols = [rng.standard_normal(n) for _ in range(8)]
    s = tuple(rng.random(ns) for _ in range(3))
    spec = CATS[cat]
    gout = [rng.standard_normal(ns) for _ in range(CatalogC(**spec).L)]
    ctx = Context(0)
    ctx.set_particles(x, y, z, m, h, rho, cols)
    ctx.build(want_perm=False)
    got = ctx.adjoint_points(*s, CatalogC(**spec), gout, strategy=strategy)
    assert ctx.lib.psb_test_adjoint_pool(ctx.h, 0, 0) == L.PSB_OK
    one = ctx.adjoint_points(*s, CatalogC(**spec), gout, strategy=strategy)
    ref = O.Oracle(x, y, z, m, h, rho, cols=cols).adjoint_points(*s, O.Catalog(**spec), gout, strategy=strategy,
                                                                hmode=O.H_NEAREST)
    for key in ("m", "x", "y", "z"):
        scale = max(np.abs(one[key]).max(), 1e-300)
        assert np.abs(got[key] - one[key]).max() <= 1e-12 * scale, key
        if ns >= 700:
            assert np.abs(got[key] - ref[key]).max() <= 1e-10 * np.abs(ref[key]).max(), key
    for a, b in zip(got["cols"], one["cols"]):
        assert np.abs(a - b).max() <= 1e-12 * max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("strategy", [L.PSB_SCATTER, L.PSB_SYMMETRIC])
@pytest.mark.parametrize("nx,ny", [(2, 2), (64, 40), (33, 130)])
def test_beam_supports_of_every_size(nx, ny, strategy):
    """Supports from a tenth of a pixel to most of the image, inside, across its
    edges and outside: a lane's, eight lanes' and a warp's particles."""
    rng = np.random.default_rng(nx)
    n = 400
    x, y, z = rng.uniform(-0.7, 0.7, n), rng.uniform(-0.7, 0.7, n), rng.uniform(-1, 1, n)
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    h = np.exp(rng.uniform(np.log(0.001), np.log(0.3), n))
    cols = [rng.standard_normal(n) for _ in range(3)]
    c, s = np.cos(0.4), np.sin(0.4)
    frame = np.array([0.05, -0.02, 0.1, c, s, 0, -s, c, 0, 0, 0, 1.0])
    prm = np.array([-0.5, 0.5, -0.4, 0.45])
    scal, shep = [0, 2], [0, 1]
    gout = [rng.standard_normal(nx * ny) for _ in scal]
    hs = np.array([0.02])
    ctx = Context(0)
    ctx.set_particles(x, y, z, m, h, rho, cols)
    ctx.build(want_perm=False)
    got = ctx.adjoint_beam(frame, prm, nx, ny, CatalogC(scalars=scal, shepard=shep), gout, strategy=strategy,
                           hmode=L.PSB_H_CONSTANT, hs=hs)
    from partia_b200 import workloads as W
    o = W.plane_coordinates(frame, (prm[0], prm[1], nx), (prm[2], prm[3], ny))
    d = tuple(np.full(nx * ny, frame[9 + k]) for k in range(3))
    ref = O.Oracle(x, y, z, m, h, rho, cols=cols).adjoint_lines(o, d, scal, gout, shepard=shep, strategy=strategy,
                                                               hmode=O.H_CONSTANT, hs=hs)
    for key in ("m", "x", "y", "z"):
        assert np.abs(got[key] - ref[key]).max() <= 1e-10 * np.abs(ref[key]).max(), key
    for k in scal:
        assert np.abs(got["cols"][k] - ref["cols"][k]).max() <= 1e-10 * np.abs(ref["cols"][k]).max(), k
