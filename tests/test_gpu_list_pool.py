"""The chunk pool of the point path's pair lists: sized by need.

 * A call on an ordinary set takes the lists and an eighth of a chunk a sample
   (65536 chunks at least).
 * A call that runs out of chunks leaves samples to the single kernel; the pool
   of the following calls holds them.  The same bits each time.
 * A refused request for list memory takes a smaller pool, and is not repeated.
 * The chunked host-memory calls, whose four sets have a pool each.
"""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

if not has_gpu():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch  # noqa: E402
from partia_b200 import _lib as L  # noqa: E402
from partia_b200.engine import CatalogC, Context  # noqa: E402

MIB = 1 << 20
SPEC = dict(scalars=[0, 1], shepard=[0, 1], grads=[-1, 1])


def context(n, seed, kid=L.PSB_KERNEL_M4):
    rng = np.random.default_rng(seed)
    x, y, z = rng.random((3, n))
    m, rho = rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.5, 2.0, n)
    h = 1.2 * n ** (-1 / 3) * rng.uniform(0.8, 1.2, n)
    ctx = Context(0)
    ctx.set_particles(x, y, z, m, h, rho, [rng.standard_normal(n) for _ in range(2)], kernel=kid)
    ctx.build(want_perm=False)
    return ctx


def scratch_of(fn):
    """MiB that a call takes and keeps."""
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    fn()
    torch.cuda.synchronize()
    return (free - torch.cuda.mem_get_info()[0]) / MIB


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
@pytest.mark.parametrize("ns", [10_000, 100_000, 1_000_000])
def test_ordinary_sets_take_little(ns, prec):
    rng = np.random.default_rng(61)
    s = [torch.tensor(a, device="cuda") for a in rng.random((3, ns))]
    out = torch.empty(ns, dtype=torch.float64, device="cuda")
    ctx = context(200_000, 60)
    dens = scratch_of(lambda: ctx.density(*s, strategy=L.PSB_GATHER, hmode=L.PSB_H_NEAREST, prec=prec, out=out))
    # a list of 32 entries of 20 bytes, h, counters and the sort's 24 bytes a sample,
    # an eighth of a chunk (32 * 20 + 16 + 9 bytes), at least 65536 in all; 8 MiB
    # for the allocator's granularity; in FP64 the particles' 48 bytes of records
    chunks = max(ns / 8, 65536)
    records = 48 * 200_000 if prec == L.PSB_PREC_FP64 else 0
    assert dens <= (ns * (640 + 13 + 32) + chunks * 665 + records) * 1.02 / MIB + 8


def dense_samples(ns, share, seed, reach=0.3):
    rng = np.random.default_rng(seed)
    s = rng.random((3, ns))
    hs = np.full(ns, 0.01)
    hs[rng.random(ns) < share] = reach
    return s, hs


@pytest.mark.parametrize("prec", [L.PSB_PREC_FP64, L.PSB_PREC_FP32C])
def test_pool_grows_to_the_need(prec):
    ns = 40_000
    ctx = context(30_000, 62)
    s, hs = dense_samples(ns, 0.2, 63)
    s = [torch.tensor(a, device="cuda") for a in s]
    hs = torch.tensor(hs, device="cuda")
    cat = CatalogC(**SPEC)
    outs = [torch.empty(ns, dtype=torch.float64, device="cuda") for _ in range(cat.L)]
    kw = dict(strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec, out=outs)
    ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
    ctx.interp_points(*s, cat, **kw)
    one, pairs = [o.clone() for o in outs], ctx.last_stats.pairs
    ctx.extra_flags = 0
    free = torch.cuda.mem_get_info()[0]
    grown = []
    for _ in range(4):
        grown.append(scratch_of(lambda: ctx.interp_points(*s, cat, **kw)))
        assert ctx.last_stats.pairs == pairs
        for a, b in zip(outs, one):
            assert torch.equal(a.nan_to_num(nan=7.0), b.nan_to_num(nan=7.0))
    assert grown[1] > 64  # the first call had too few chunks
    assert grown[2] + grown[3] <= 64, grown  # and the second enough, or nearly
    assert sum(grown[1:]) * MIB <= free / 16


def test_refused_list_memory():
    ns = 40_000
    ctx = context(30_000, 64)
    s, hs = dense_samples(ns, 0.2, 65)
    kw = dict(strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs)
    first = ctx.density(*s, **kw)  # runs out; asks for more
    assert ctx.lib.psb_test_list_pool(ctx.h, 0, 1) == L.PSB_OK
    free = torch.cuda.mem_get_info()[0]
    assert np.array_equal(ctx.density(*s, **kw), first)  # refused: the first call's pool
    assert np.array_equal(ctx.density(*s, **kw), first)  # (and no more asked for)
    assert torch.cuda.mem_get_info()[0] >= free - 8 * MIB

    ctx = context(30_000, 64)
    assert ctx.lib.psb_test_list_pool(ctx.h, 0, 1) == L.PSB_OK
    assert np.array_equal(ctx.density(*s, **kw), first)  # the least pool
    assert np.array_equal(ctx.density(*s, **kw), first)
    assert ctx.lib.psb_test_list_pool(ctx.h, 0, 1) == L.PSB_OK
    with pytest.raises(L.PsbError) as e:  # not even that
        ctx.density(*s, **kw)
    assert e.value.code == L.PSB_ENOMEM
    assert np.array_equal(ctx.density(*s, **kw), first)
    for chunks in (1, 33, 5000):  # a pool of any size: the same bits
        assert ctx.lib.psb_test_list_pool(ctx.h, chunks, 0) == L.PSB_OK
        assert np.array_equal(ctx.density(*s, **kw), first)


@pytest.mark.parametrize("kid,prec", [(L.PSB_KERNEL_M4, L.PSB_PREC_FP32C), (L.PSB_KERNEL_M6, L.PSB_PREC_FP32C),
                                      (L.PSB_KERNEL_M5, L.PSB_PREC_FP64)])
def test_chunked_host_calls_with_large_neighbourhoods(kid, prec):
    """Host arrays of more than 2^20 samples go in chunks through four sets of
    lists, with a pool each that runs out in the first call."""
    ns = (1 << 20) + 12_345
    ctx = context(30_000, 66, kid)
    s, hs = dense_samples(ns, 0.02, 67, 0.2)
    cat = CatalogC(scalars=[0, 1], shepard=[0, 1], grads=[1])
    kw = dict(strategy=L.PSB_GATHER, hmode=L.PSB_H_PER_SAMPLE, hs=hs, prec=prec)
    ctx.extra_flags = L.PSB_FLAG_SINGLE_KERNEL
    one = ctx.interp_points(*s, cat, **kw)
    pairs = ctx.last_stats.pairs
    ctx.extra_flags = 0
    for _ in range(3):
        got = ctx.interp_points(*s, cat, **kw)
        assert ctx.last_stats.pairs == pairs
        for a, b in zip(got, one):
            assert np.array_equal(a, b, equal_nan=True)
