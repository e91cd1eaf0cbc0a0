"""The FP64 pair sums' leaf records: filled by the first FP64 call after a build,
of sets of up to 2^20 particles by the build.

Contexts of larger sets that only run FP32C hold none; results do not depend on
when they were filled, nor on whether a call found them (the call that may not
allocate).
"""
import ctypes as C

import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if not has_gpu():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch  # noqa: E402
from partia_b200 import _lib as L  # noqa: E402
from partia_b200.engine import CatalogC, Context  # noqa: E402

SPEC = dict(scalars=[0, 1], shepard=[0, 1], grads=[-1, 1])


def arrays(n, seed, dtype=np.float64):
    rng = np.random.default_rng(seed)
    x, y, z = rng.random((3, n))
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    h = 1.2 * n ** (-1 / 3) * rng.uniform(0.8, 1.2, n)
    return [a.astype(dtype) for a in (x, y, z, m, h, rho)], [rng.standard_normal(n).astype(dtype) for _ in range(2)]


def test_only_fp64_calls_hold_them():
    n, ns = 2_000_000, 1000
    arrs, cols = arrays(n, 81)
    s = [torch.tensor(a, device="cuda") for a in np.random.default_rng(82).random((3, ns))]
    out = torch.empty(ns, dtype=torch.float64, device="cuda")
    ctx = Context(0)
    ctx.set_particles(*arrs, cols=cols)
    ctx.build(want_perm=False)
    kw = dict(strategy=L.PSB_SCATTER, out=out)
    free = []
    for prec in (L.PSB_PREC_FP32C, L.PSB_PREC_FP32C, L.PSB_PREC_FP64):
        ctx.density(*s, prec=prec, **kw)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[1] - free[2] >= 47 * n  # 48 bytes a particle, not before the FP64 call


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [20_000, 1_100_000])
@pytest.mark.parametrize("kid", [L.PSB_KERNEL_M4, L.PSB_KERNEL_C2])
def test_results_do_not_depend_on_when_they_were_filled(n, kid, dtype):
    ns = 3000
    arrs, cols = arrays(n, 83, dtype)
    rng = np.random.default_rng(84)
    s = [torch.tensor(a.astype(dtype), device="cuda") for a in rng.random((3, ns))]
    cat = CatalogC(**SPEC)
    outs = [torch.empty(ns, dtype=s[0].dtype, device="cuda") for _ in range(cat.L)]
    kw = dict(strategy=L.PSB_SYMMETRIC, out=outs)

    def fields(ctx, **k):
        ctx.interp_points(*s, cat, **kw, **k)
        return [o.clone() for o in outs]

    def equal(a, b):
        return all(torch.equal(u.nan_to_num(nan=7.0), v.nan_to_num(nan=7.0)) for u, v in zip(a, b))

    def without(ctx):  # the call that may not allocate
        ptrs = (C.c_void_p * cat.L)(*[o.data_ptr() for o in outs])
        rc = ctx.lib.psb_interp_points_noalloc(ctx.h, ns, *[a.data_ptr() for a in s], L.PSB_H_NEAREST, None,
                                               L.PSB_SYMMETRIC, C.byref(cat.c), L.PSB_PREC_FP64, ptrs, None)
        assert rc == L.PSB_OK
        return [o.clone() for o in outs]

    ctx = Context(0)
    ctx.set_particles(*arrs, cols=cols, kernel=kid)
    perm, *_ = ctx.build()
    bare = without(ctx)  # no records yet, of the larger sets
    first = fields(ctx)
    held = without(ctx)  # with them
    assert equal(bare, held)
    if dtype == np.float64:
        assert equal(first, bare)
    # new values: the held records follow
    m2, rho2 = arrs[3] * dtype(1.5), arrs[5] * dtype(0.75)
    ctx.set_values(m2[perm], rho2[perm], [c[perm] for c in cols])
    new = fields(ctx)
    other = Context(0)
    other.set_particles(*arrs, cols=cols, kernel=kid)
    other.build(want_perm=False)
    other.set_values(m2[perm], rho2[perm], [c[perm] for c in cols])
    assert equal(fields(other), new) and not equal(new, first)
    # another set in the same context
    arrs3, cols3 = arrays(n // 2, 85, dtype)
    for c in (ctx, other):
        c.set_particles(*arrs3, cols=cols3, kernel=kid)
        c.build(want_perm=False)
    fields(other, prec=L.PSB_PREC_FP32C)
    assert equal(fields(ctx), fields(other))
