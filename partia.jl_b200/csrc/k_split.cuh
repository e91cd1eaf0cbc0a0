// k_split.cuh -- the point path over pair lists: walk, then sums.
//
// k_collect walks the LBVH for a tile of 32 samples (one warp, 32 nodes a step,
// with the spans and inclusion decisions of k_points) and records, per sample,
// the accepted leaves as one entry per span (first leaf, 32-bit mask, the
// sample's offset from the first leaf) plus the sample's smoothing length.  It
// keeps no accumulators, so it runs with few registers.
// k_bodies then evaluates the kernel weights and sums of every recorded pair:
// each lane runs through a list part (a sample's list in its tile, or one of
// its chunks) in one flattened loop, so a warp iteration does 32 pair bodies
// until the shortest parts run out, instead of idling lanes once per span.
// Pairs are visited in the same order as in k_points (span order, then leaf
// order), with the same arithmetic.
#pragma once

#include "k_points.cuh"

namespace psb {

constexpr int BODY_THREADS = 128, WALK_THREADS = 128;  // threads of a block of the pair sums and of the walk

// Per-warp shared memory of the walk.
constexpr int WQ = 192;  // stack of the walk
// Two leaves' negated positions (relative to the warp anchor for double inputs,
// as they are for float ones) and squared radii: one packed operation takes
// both leaves.
struct LeafPair {
    float2 x, y, z, T;
};
struct CStage {
    LeafPair L[SPAN / 2];
    float4 P[SPAN];   // samples: position as the leaves', squared radius or nearest candidate bound
    float4 W[SPAN];   // samples: float position and squared radius bound, for node tests one by one
    int32_t q[WQ];
    // leaf j of the span (all 32 lanes call; a last odd leaf is paired with one out of reach)
    __device__ __forceinline__ void put(int j, int cnt, float x, float y, float z, float T) {
        if (j < cnt || j == cnt) {
            const bool pad = j == cnt;
            if (pad && !(cnt & 1)) return;
            float* o = (float*)&L[j >> 1] + (j & 1);
            o[0] = pad ? 1e18f : -x;
            o[2] = pad ? 1e18f : -y;
            o[4] = pad ? 1e18f : -z;
            o[6] = pad ? 0.f : T;
        }
    }
};
// The walk in the particles' own arithmetic (WIDE): the samples, each with its
// squared radius or nearest candidate distance (below 0: takes no part).
template <class T> struct WStage : CStage {
    T wx[SPAN], wy[SPAN], wz[SPAN], wr2[SPAN];
    T lx[SPAN], ly[SPAN], lz[SPAN], lr2[SPAN];  // the span's leaves
};
__device__ __forceinline__ uint64_t pk(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpk(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// Squared distances of a sample (x, y, z packed twice) from a pair of leaves:
// fused for the float tests, in the reference's operation order (EXACT) for
// float inputs.
template <bool EXACT>
__device__ __forceinline__ float2 pair_d2(uint64_t px, uint64_t py, uint64_t pz, const LeafPair& q) {
    const uint64_t dx = add2(px, pk(q.x.x, q.x.y)), dy = add2(py, pk(q.y.x, q.y.y)), dz = add2(pz, pk(q.z.x, q.z.y));
    if (EXACT) {
        // the products one by one: a packed product may be merged into the packed sum behind it
        const float2 x = unpk(dx), y = unpk(dy), z = unpk(dz);
        const uint64_t xx = pk(__fmul_rn(x.x, x.x), __fmul_rn(x.y, x.y)), yy = pk(__fmul_rn(y.x, y.x), __fmul_rn(y.y, y.y)),
                       zz = pk(__fmul_rn(z.x, z.x), __fmul_rn(z.y, z.y));
        return unpk(add2(add2(xx, yy), zz));
    }
    return unpk(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, 0ull))));
}
// v's sign bit shifted into m from below
__device__ __forceinline__ unsigned push_sign(unsigned m, float v) { return __funnelshift_l(__float_as_uint(v), m, 1); }
// found spans that reached none of the warp's samples, after which its node
// tests go sample by sample
constexpr int WALK_MISSES = 12;

// A sample's list part is full: start its next one.  Takes a chunk of the
// pool, or after HEAVY_PARTS parts hands the sample to k_heavy, as long as its
// list has room.  Returns the sample's current chunk and its parts: parts = 0
// if it is k_heavy's, unchanged if the pool has run out.
static __device__ __noinline__ int2 next_part(const SplitBufs& sp, uint32_t idx, int32_t chunk, int nparts) {
    if (nparts == HEAVY_PARTS) {
        const unsigned slot = atomicAdd(sp.hcount, 1u);
        if (slot < sp.hcap) {
            sp.hlist[slot] = idx;
            return make_int2(chunk, 0);
        }
    }
    const unsigned c = atomicAdd(sp.top, 1u);
    if (c >= sp.ncap) return make_int2(chunk, nparts);
    if (chunk >= 0) {
        sp.next[chunk] = (int32_t)c;
        sp.ccnt[chunk] = (uint8_t)RCAP;
    } else {
        sp.head[idx] = (int32_t)c;
    }
    sp.own[c] = idx | (chunk >= 0 ? OWN_LATER : 0u);
    if (chunk < 0 && sp.mlist) sp.mlist[atomicAdd(sp.mcount, 1u)] = c;
    return make_int2((int32_t)c, nparts + 1);
}

// Samples left to the single kernel (their cnt is CNT_DEAD): their tile is
// listed once, by whoever marks the first of its samples.
static __device__ __forceinline__ void list_dead(const SplitBufs& sp, uint32_t bt, unsigned mask) {
    if (atomicOr(&sp.dead[bt], mask) == 0u) sp.ovf_tiles[atomicAdd(sp.ovf_count, 1u)] = (int32_t)(sp.tile0 + bt);
}

// The walk of one warp: the nodes that reach the warp's samples, found 32 at a
// time.  The stack holds nodes (id) and found spans (-id) with the leftmost
// item on top.  A step takes the top items of the stack, one per lane, tests
// the nodes against the box around the samples, and puts the survivors'
// children back where the nodes were (a subtree of at most SPAN leaves as a
// found span), so the spans come off the top in leaf order.  The union walk
// of 32 samples that tested one node a step took as many dependent loads as
// it visited nodes; here a step's loads are independent and a walk takes a
// few more steps than the tree has levels.  ORDERED = false hands out the spans as
// they come (the nearest search, whose bound they tighten).
// node_ok(ni): whether internal node ni may hold something; span_fn(id) is
// called by all lanes.  Corrupt links end the walk with an error: the links
// are those the escape-link walks use, so a tree whose root has an escape (it
// has none) is refused, and steps and stack are bounded.
template <bool ORDERED, class T, class NodeOk, class SpanFn>
__device__ __forceinline__ bool window_walk(const TreeView<T>& tv, int32_t* q, NodeOk node_ok, SpanFn span_fn,
                                            uint32_t& steps) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int32_t n = (int32_t)tv.n;
    if (tv.root == 0) {  // a single particle
        span_fn(n);
        return true;
    }
    if (__ldg(&tv.links[tv.root - 1]).y != 0) return false;
    __syncwarp();
    if (lane == 0) q[0] = tv.root;
    __syncwarp();
    int top = 1;
    const uint32_t bound = (uint32_t)(4 * tv.n + 8 < 0xFFFFFFFFll ? 4 * tv.n + 8 : 0xFFFFFFFFll);
    uint32_t k = 0;
    while (top > 0) {
        if (++k >= bound) return false;
        // near the stack's end the window narrows to one node: depth first, one item a level
        const int w = min(32, min(top, max(1, WQ - 64 - top)));
        const int32_t id = lane < w ? q[top - 1 - lane] : 0;
        const unsigned spans = __ballot_sync(PSB_FULL, id < 0);
        if (ORDERED) {
            const int lead = __ffs(~spans) - 1;  // spans on top (-1: all 32)
            if (spans & 1u) {
                const int m = lead < 0 ? 32 : lead;
                top -= m;
                for (int c = 0; c < m; ++c) span_fn(-__shfl_sync(PSB_FULL, id, c));
                continue;
            }
        }
        int out = 0;
        int32_t c0 = 0, c1 = 0;
        if (id < 0) {
            out = ORDERED ? 1 : 0;
            c0 = id;
        } else if (id >= n) {  // a leaf reached directly: a span of one
            out = 1;
            c0 = -id;
        } else if (id > 0) {
            const int4 lk = __ldg(&tv.links[id - 1]);
            if (node_ok(id - 1)) {
                if (lk.w - lk.z < SPAN) {
                    out = 1;
                    c0 = -id;
                } else {
                    out = 2;
                    c0 = lk.x;
                    c1 = __ldg(&tv.right[id - 1]);
                }
            }
        }
        const unsigned b1 = __ballot_sync(PSB_FULL, out == 1), b2 = __ballot_sync(PSB_FULL, out == 2);
        top += __popc(b1) + 2 * __popc(b2) - w;
        if (top > WQ) return false;
        const int at = top - 1 - __popc(b1 & below) - 2 * __popc(b2 & below);
        __syncwarp();
        if (out) q[at] = c0;
        if (out == 2) q[at - 1] = c1;
        __syncwarp();
        if (!ORDERED)
            for (unsigned m = spans; m; m &= m - 1) span_fn(-__shfl_sync(PSB_FULL, id, __ffs(m) - 1));
    }
    steps += k;
    return true;
}

// The pair lists of a tile's samples (or, in a call of few samples, of
// 2^lspt of them, so that the call has enough warps): the nearest particle's
// h where it is asked for, then every leaf within the support radii.
// Node tests are conservative in float (records rounded outwards) against the
// box around the samples; a span is then tested against each sample, and its
// leaves decided as k_points decides them.
//
// Bound by issue (compare and vote work of the span tests) on full grids, by
// the longest walk in small calls.  10 CTAs (40 warps) per SM: 8 / 10 / 12 CTAs
// take 4.75 / 4.68 / 4.78 ms on the 2M-particle 128^3 grid (FP32C, 8 fields)
// and 2.79 / 2.72 / 2.82 ms on 700k unordered points.  Before, with one node a
// step: 5.45 and 2.97 ms; FP64 on 500k particles and a 101 x 67 x 53 grid,
// which walked in double, 4.05 -> 1.66 ms; 37 points 4.7 -> 0.37 ms.  The leaf
// tests then took two leaves an instruction, the sign of d^2 - r^2 as the
// decision and one tolerance per span, in place of two thresholds compared per
// leaf: 4.70 -> 4.49 ms (FP32C), 1.66 -> 1.40 ms (FP64).
//
// WIDE: particle sets outside the float tests' range (psb_ctx::band_ok), with
// every test in the reference's arithmetic.  Differences, squares and their sums
// round monotonically, so the box around the samples is nearer to a node than any
// of them, and a node than its leaves, in that arithmetic too: no margins.
// 1M uniform particles, 96^3 grid, FP64 at 4e20: gather 4.5 -> 2.5 ms, symmetric
// 4.9 -> 2.7 (the single kernel took such sets; in the float tests' range 1.7, 1.8).
template <class T, int ST, bool WIDE>
__global__ void __launch_bounds__(WALK_THREADS, (WIDE ? 640 : 1280) / WALK_THREADS)
    k_collect(const __grid_constant__ Args<T> A) {
    constexpr bool BAND = sizeof(T) == 8;
    __shared__ typename std::conditional<WIDE, WStage<T>, CStage>::type stage_all[WALK_THREADS / 32];
    const TreeView<T>& tv = A.tv;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    auto& st = stage_all[wib];
    const int lspt = A.sp.lspt;
    const int64_t wid = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    const int64_t bt = wid >> (5 - lspt);
    if (bt >= A.sp.ntiles) return;  // warp-uniform
    const int64_t tile = A.sp.tile0 + bt;
    // this warp's samples: lanes 0 .. 2^lspt - 1 take the tile's samples slot
    const int s0 = ((int)wid & ((32 >> lspt) - 1)) << lspt;
    const bool mine = lane < (1 << lspt);
    const uint32_t slot = (uint32_t)(bt * 32) + (uint32_t)(s0 + (mine ? lane : 0));

    const int64_t k = mine ? sample_of(A.src, tile, s0 + lane) : -1;
    const bool valid = k >= 0;
    T p[3] = {T(0), T(0), T(0)}, dd[3];
    if (valid) sample_coords(A.src, k, p, dd);
    // A sample whose position or h is not finite, or (not WIDE) beyond the range of
    // the float tests, sends its warp's samples to the single kernel.
    {
        constexpr double most = WIDE ? 1.7976931348623157e308 : 1e18;
        bool wild = valid && !(fabs((double)p[0]) <= most && fabs((double)p[1]) <= most && fabs((double)p[2]) <= most);
        if (ST != ST_SCATTER && A.hmode != PSB_H_NEAREST && valid)
            wild = wild || !(fabs((double)((A.hmode == PSB_H_PER_SAMPLE) ? A.hs[k] : A.hs[0])) <= most);
        const bool any_wild = __any_sync(PSB_FULL, wild);
        if (any_wild || !__any_sync(PSB_FULL, valid)) {
            if (mine) {
                A.sp.cnt[slot] = any_wild ? CNT_DEAD : 0;
                A.sp.head[slot] = -1;
            }
            if (any_wild && lane == 0) list_dead(A.sp, (uint32_t)bt, 0xffffffffu >> (32 - (1 << lspt)) << s0);
            return;
        }
    }
    uint32_t n_pairs = 0, n_retest = 0, n_spans = 0, n_parts = 0;  // per lane / warp, widened below
    uint32_t steps = 0;
    bool ok = true;

    // the box around the warp's samples (float, rounded outwards)
    float blo[3], bhi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float a = valid ? __double2float_rd((double)p[d]) : INFINITY, b = valid ? __double2float_ru((double)p[d]) : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a = fminf(a, __shfl_xor_sync(PSB_FULL, a, o));
            b = fmaxf(b, __shfl_xor_sync(PSB_FULL, b, o));
        }
        blo[d] = a;
        bhi[d] = b;
    }
    // lower bound of the squared distance between that box and a node's
    auto box_d2 = [&](const float4& lo, const float4& hi) -> float {
        const float tx = fmaxf(fmaxf(lo.x - bhi[0], blo[0] - hi.x), 0.f);
        const float ty = fmaxf(fmaxf(lo.y - bhi[1], blo[1] - hi.y), 0.f);
        const float tz = fmaxf(fmaxf(lo.z - bhi[2], blo[2] - hi.z), 0.f);
        return (tx * tx + ty * ty + tz * tz) * (1.f - RELM);
    };
    const float pf[3] = {(float)p[0], (float)p[1], (float)p[2]};
    const float pem = U1 * fmaxf(fmaxf(fabsf(pf[0]), fabsf(pf[1])), fabsf(pf[2])) + 1e-30f;
    // The box test serves samples close to one another.  Where they are not (a
    // tile across a jump of the Morton curve, one sample of a far larger
    // radius), the box reaches nodes that no sample does: after WALK_MISSES
    // such spans a node must also reach one of the samples themselves.
    int misses = 0;  // warp-uniform
    const float pemx = __uint_as_float(__reduce_max_sync(PSB_FULL, valid ? __float_as_uint(pem) : 0u));
    auto set_sample = [&](bool on, float r2) { st.W[lane] = make_float4(on ? pf[0] : 1e30f, pf[1], pf[2], r2); };
    auto any_sample = [&](const float4& lo, const float4& hi, float r2n) -> bool {
        for (int s = 0; s < (1 << lspt); ++s) {
            const float4 w = st.W[s];
            const float q[3] = {w.x, w.y, w.z};
            // (a node whose h is NaN is not left out by it: the box test's answer)
            if (!(lb_d2_pbox(q, pemx, lo, hi) > (ST == ST_SCATTER ? r2n : fmaxf(w.w, r2n)))) return true;
        }
        return false;
    };

    // WIDE: the samples as they are, the box around them, and the exact squared
    // distance of that box, and of the samples, from node ni
    T lob[3] = {T(0), T(0), T(0)}, hib[3] = {T(0), T(0), T(0)};
    auto wide_max = [&](T v) -> T {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const T u = __shfl_xor_sync(PSB_FULL, v, o);
            v = u > v ? u : v;
        }
        return v;
    };
    if constexpr (WIDE) {
        st.wx[lane] = p[0]; st.wy[lane] = p[1]; st.wz[lane] = p[2];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lob[d] = -wide_max(valid ? -p[d] : -(T)INFINITY);
            hib[d] = wide_max(valid ? p[d] : -(T)INFINITY);
        }
    }
    auto wide_box_d2 = [&](int ni) -> T {
        T r = T(0);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const T a = __ldg(&tv.nmin[d][ni]), b = __ldg(&tv.nmax[d][ni]);
            const T t = hib[d] < a ? X<T>::sub(a, hib[d]) : (lob[d] > b ? X<T>::sub(lob[d], b) : T(0));
            r = X<T>::add(r, X<T>::mul(t, t));
        }
        return r;
    };
    auto wide_any = [&](int ni, bool near) -> bool {
        if constexpr (WIDE) {
            const T hn = ST == ST_GATHER || near ? T(0) : __ldg(&tv.nscale[ni]);
            for (int s = 0; s < (1 << lspt); ++s) {
                const T r2 = st.wr2[s];
                const T q[3] = {st.wx[s], st.wy[s], st.wz[s]};
                if (r2 >= T(0) && !(ex_d2_pbox<T>(q, tv, ni) > (near ? r2 : ex_r2<ST, T>(r2, hn, (T)tv.Kd)))) return true;
            }
        }
        return false;
    };
    // The leaves of the span within a taking sample's radius, the particle's
    // (SA = ST_SCATTER), or the larger one, by the loop with fewer tests.
    auto wide_leaves = [&](int64_t lo, int cnt, unsigned parts, auto sa) -> unsigned {
        unsigned mine = 0;
        if constexpr (WIDE) {
            constexpr int SA = decltype(sa)::value;
            auto radius = [&](T r2s, T r2b) { return SA == ST_GATHER ? r2s : (SA == ST_SCATTER ? r2b : jmax(r2s, r2b)); };
            const bool by_sample = __popc(parts) >= cnt;
            T lx = T(0), ly = T(0), lz = T(0), r2b = T(0);
            if (lane < cnt) {
                lx = __ldg(&tv.x[lo + lane]); ly = __ldg(&tv.y[lo + lane]); lz = __ldg(&tv.z[lo + lane]);
                if (SA != ST_GATHER) r2b = ex_r2<ST_SCATTER, T>(T(0), __ldg(&tv.h[lo + lane]), (T)tv.Kd);
            }
            __syncwarp();
            if (by_sample) {
                st.lx[lane] = lx; st.ly[lane] = ly; st.lz[lane] = lz; st.lr2[lane] = r2b;
                __syncwarp();
                if ((parts >> lane) & 1u) {
                    const T r2s = st.wr2[lane];
#pragma unroll 4
                    for (int j = 0; j < cnt; ++j)
                        mine |= (unsigned)(ex_d2_pp<T>(p, st.lx[j], st.ly[j], st.lz[j]) <= radius(r2s, st.lr2[j])) << j;
                }
            } else {
                for (unsigned pp = parts; pp; pp &= pp - 1) {
                    const int s = __ffs(pp) - 1;
                    const T q[3] = {st.wx[s], st.wy[s], st.wz[s]};
                    const unsigned b = __ballot_sync(PSB_FULL, lane < cnt && ex_d2_pp<T>(q, lx, ly, lz) <= radius(st.wr2[s], r2b));
                    if (lane == s) mine = b;
                }
            }
            __syncwarp();
        }
        return mine;
    };

    // the warp anchor (its first sample) and the samples relative to it
    const int first = __ffs(__ballot_sync(PSB_FULL, valid)) - 1;
    const double cw[3] = {__shfl_sync(PSB_FULL, (double)p[0], first), __shfl_sync(PSB_FULL, (double)p[1], first),
                          __shfl_sync(PSB_FULL, (double)p[2], first)};
    float esmax = 0.f;  // largest error of a relative sample position
    if constexpr (BAND) {
        const float sr[3] = {(float)((double)p[0] - cw[0]), (float)((double)p[1] - cw[1]), (float)((double)p[2] - cw[2])};
        st.P[lane] = make_float4(sr[0], sr[1], sr[2], 0.f);
        if (valid) esmax = U1 * (fabsf(sr[0]) + fabsf(sr[1]) + fabsf(sr[2])) + 1e-30f;
        esmax = __uint_as_float(__reduce_max_sync(PSB_FULL, __float_as_uint(esmax)));
    } else {
        st.P[lane] = make_float4(pf[0], pf[1], pf[2], 0.f);
    }
    // the span of node id: first leaf and leaf count
    auto span_of = [&](int32_t id, int64_t& lo, int& cnt) {
        if (id >= (int32_t)tv.n) {
            lo = (int64_t)id - tv.n;
            cnt = 1;
        } else {
            const int4 lk = __ldg(&tv.links[id - 1]);
            lo = (int64_t)lk.z - 1;
            cnt = lk.w - lk.z + 1;
        }
    };
    // the span's anchor (first leaf) relative to the warp anchor, and the
    // error bound of its leaves' relative positions (the same for every leaf)
    auto anchor = [&](int64_t lo, float o[3], float lmax) -> float {
        o[0] = (float)((double)__ldg(&tv.x[lo]) - cw[0]);
        o[1] = (float)((double)__ldg(&tv.y[lo]) - cw[1]);
        o[2] = (float)((double)__ldg(&tv.z[lo]) - cw[2]);
        return U1 * (2.f * lmax + 2.f * (fabsf(o[0]) + fabsf(o[1]) + fabsf(o[2]))) * (1.f + 4.f * U1);
    };

    T ha = T(0);
    if (ST != ST_SCATTER) {
        if (A.hmode == PSB_H_NEAREST) {
            // LBVH_find_nearest_h (LinearBVHQueries.jl:118-140), see nearest_h_pass
            double best = INFINITY;
            int32_t bidx = -1;
            if (valid) nearest_seed<T>(tv, p, best, bidx);
            float bestf = __double2float_ru(best);
            set_sample(valid, bestf);
            float bmax = __uint_as_float(__reduce_max_sync(PSB_FULL, valid ? __float_as_uint(bestf) : 0u));
            T bwide = T(0);  // WIDE: the largest candidate distance (best is one in T)
            auto set_wide = [&]() {
                if constexpr (WIDE) {
                    __syncwarp();
                    st.wr2[lane] = valid ? (T)best : T(-1);
                    bwide = wide_max(valid ? (T)best : T(-1));
                    __syncwarp();
                }
            };
            set_wide();
            auto node_ok = [&](int ni) -> bool {
                if constexpr (WIDE) return !(wide_box_d2(ni) > bwide) && (misses < WALK_MISSES || wide_any(ni, true));
                const float4 lo = __ldg(&tv.node_lo[ni]), hi = __ldg(&tv.node_hi[ni]);
                return !(box_d2(lo, hi) > bmax) && (misses < WALK_MISSES || any_sample(lo, hi, 0.f));
            };
            auto span_fn = [&](int32_t id) {
                bool part = valid;
                if (WIDE && id < (int32_t)tv.n)
                    part = part && !(ex_d2_pbox<T>(p, tv, id - 1) > (T)best);
                else if (id < (int32_t)tv.n)
                    part = part && !(lb_d2_pbox(pf, pem, __ldg(&tv.node_lo[id - 1]), __ldg(&tv.node_hi[id - 1])) > bestf);
                const unsigned parts = __ballot_sync(PSB_FULL, part);
                if (!parts) {
                    ++misses;
                    return;
                }
                int64_t lo;
                int cnt;
                span_of(id, lo, cnt);
                if constexpr (WIDE) {
                    for (unsigned u = wide_leaves(lo, cnt, parts, std::integral_constant<int, ST_GATHER>()); u; u &= u - 1) {
                        const int64_t li = lo + __ffs(u) - 1;
                        const double d2 = (double)ex_d2_pp<T>(p, tv.x[li], tv.y[li], tv.z[li]);
                        if (d2 < best || (d2 == best && li < bidx)) { best = d2; bidx = (int32_t)li; }
                    }
                    set_wide();
                    return;
                }
                // candidates: float d2 not above (sqrt(best) + error)^2, or exactly not above best
                float thr;
                float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < cnt) L = __ldg(&tv.leaf4[lo + lane]);
                if constexpr (BAND) {
                    float o[3];
                    const float eqm = anchor(lo, o, __ldg(&tv.spanb[lo]).x);
                    const float bs = (float)sqrt(best);
                    const float e = 1.7320508f * (esmax + eqm) + 4.f * U1 * bs + 1e-18f;
                    const float t = (bs + e) * (1.f + 4.f * U1);
                    thr = isinf(best) ? INFINITY : t * t;
                    L.x += o[0]; L.y += o[1]; L.z += o[2];
                } else {
                    thr = (float)best;  // a float distance: exact
                }
                const bool by_sample = 3 * __popc(parts) >= 2 * cnt;
                unsigned cand = 0;
                __syncwarp();
                if (by_sample) {  // each taking lane tests its sample against every leaf
                    st.put(lane, cnt, L.x, L.y, L.z, 0.f);
                    __syncwarp();
                    if (part) {
                        const float4 P = st.P[lane];
                        const uint64_t px = pk(P.x, P.x), py = pk(P.y, P.y), pz = pk(P.z, P.z);
                        unsigned out = 0;
#pragma unroll 2
                        for (int j = (cnt - 1) >> 1; j >= 0; --j) {
                            const float2 d2 = pair_d2<!BAND>(px, py, pz, st.L[j]);
                            out = push_sign(push_sign(out, thr - d2.y), thr - d2.x);
                        }
                        cand = ~out & (0xffffffffu >> (32 - cnt));
                    }
                } else {  // lane j tests leaf j against each taking sample
                    st.P[lane].w = thr;
                    __syncwarp();
                    for (unsigned pp = parts; pp; pp &= pp - 1) {
                        const int s = __ffs(pp) - 1;
                        const float4 P = st.P[s];
                        const float dx = P.x - L.x, dy = P.y - L.y, dz = P.z - L.z;
                        float d2;
                        if constexpr (BAND) d2 = dx * dx + dy * dy + dz * dz;
                        else d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                        const unsigned b = __ballot_sync(PSB_FULL, lane < cnt && d2 <= P.w);
                        if (lane == s) cand = b;
                    }
                }
                for (; cand; cand &= cand - 1) {
                    const int64_t li = lo + __ffs(cand) - 1;
                    const double d2 = (double)ex_d2_pp<T>(p, tv.x[li], tv.y[li], tv.z[li]);
                    if (d2 < best || (d2 == best && li < bidx)) { best = d2; bidx = (int32_t)li; bestf = __double2float_ru(best); }
                }
                st.W[lane].w = bestf;
                bmax = __uint_as_float(__reduce_max_sync(PSB_FULL, valid ? __float_as_uint(bestf) : 0u));
            };
            ok = window_walk<false>(tv, st.q, node_ok, span_fn, steps);
            ha = valid ? ((bidx >= 0) ? tv.h[bidx] : qnan<T>()) : T(0);
        } else if (valid) {
            ha = (A.hmode == PSB_H_PER_SAMPLE) ? A.hs[k] : A.hs[0];
        }
    }
    const T Kt = (T)tv.Kd;
    const T ra = X<T>::mul(Kt, ha);
    const T ra2 = X<T>::mul(ra, ra);
    // a sample of radius NaN (the nearest particle's h, or none near) has no
    // neighbours, in the symmetric strategy either (jmax(NaN, r) is NaN)
    const bool takes = valid && (ST == ST_SCATTER || ra2 == ra2);
    float ra2_hi = 0.f, rahi = 0.f;
    if (ST != ST_SCATTER) {
        rahi = __double2float_ru(fabs((double)ra)) * (1.f + 2.f * U1);
        ra2_hi = takes ? __double2float_ru((double)ra2) * (1.f + RELM) + 1e-36f : 0.f;
    }
    // tile-wide maxima (NaN reaches nothing)
    auto warp_max = [&](float v) { return __uint_as_float(__reduce_max_sync(PSB_FULL, v > 0.f ? __float_as_uint(v) : 0u)); };
    const float rahimax = warp_max(rahi);
    float ra2max = warp_max(ra2_hi);
    misses = 0;
    __syncwarp();
    set_sample(takes, ra2_hi);
    const T ra2w = !takes ? T(-1) : (ST == ST_SCATTER ? T(0) : ra2);
    T ra2wmax = T(-1);  // WIDE: the largest squared radius
    if constexpr (WIDE) {
        st.wr2[lane] = ra2w;
        ra2wmax = wide_max(ra2w);
        __syncwarp();
    }

    // this lane's pair list: the next entry goes to index epos
    uint32_t epos = (uint32_t)bt * (RCAP * 32) + (slot & 31);
    int nent = 0;         // entries in the current part
    int32_t chunk = -1;   // the current chunk (-1: the tile's list)
    int nparts = 1;       // parts so far; 0: the sample is k_heavy's
    bool dead = false;    // warp-uniform: the pool ran out, the samples are k_points'
    auto emit = [&](int64_t lo, unsigned acc) {
        if (__any_sync(PSB_FULL, acc && nent == RCAP)) {
            if (acc && nent == RCAP) {
                const int2 q = next_part(A.sp, slot, chunk, nparts);
                if (q.y > nparts) {
                    chunk = q.x;
                    epos = A.sp.ebase + (uint32_t)chunk * RCAP;
                    nent = 0;
                }
                nparts = q.y;
            }
            if (nparts == 0) {
                acc = 0;
                ra2_hi = 0.f;
                st.W[lane].x = 1e30f;
                if constexpr (WIDE) st.wr2[lane] = T(-1);
            }
            dead = __any_sync(PSB_FULL, acc && nent == RCAP);
            if (ST == ST_GATHER) {  // (the other strategies reach nodes by h_b too)
                if constexpr (WIDE) ra2wmax = wide_max(nparts > 0 ? ra2w : T(-1));
                else ra2max = warp_max(ra2_hi);
            }
        }
        if (!acc || dead) return;
        n_pairs += __popc(acc);
        // the sample relative to the span's first leaf, in double then
        // rounded: the pair separation R - L carries only the rounding of
        // two small vectors
        float r0 = 0.f, r1 = 0.f, r2 = 0.f;
        if (BAND && !A.sp.fp64) {
            r0 = (float)((double)p[0] - (double)__ldg(&tv.x[lo]));
            r1 = (float)((double)p[1] - (double)__ldg(&tv.y[lo]));
            r2 = (float)((double)p[2] - (double)__ldg(&tv.z[lo]));
        }
        A.sp.ent4[epos] = make_float4(r0, r1, r2, __int_as_float((int)lo));
        A.sp.emask[epos] = acc;
        epos += chunk >= 0 ? 1 : 32;
        ++nent;
    };

    auto node_ok = [&](int ni) -> bool {
        if (dead) return false;
        if constexpr (WIDE) {
            const T r2 = ST == ST_GATHER ? ra2wmax : ex_r2<ST, T>(ra2wmax, __ldg(&tv.nscale[ni]), Kt);
            return !(wide_box_d2(ni) > r2) && (misses < WALK_MISSES || wide_any(ni, false));
        }
        const float4 lo = __ldg(&tv.node_lo[ni]), hi = __ldg(&tv.node_hi[ni]);
        if (box_d2(lo, hi) > hi_r2_node<ST>(ra2max, lo.w, tv.Kf)) return false;
        return misses < WALK_MISSES || any_sample(lo, hi, ST == ST_GATHER ? 0.f : hi_r2_node<ST_SCATTER>(0.f, lo.w, tv.Kf));
    };
    auto span_fn = [&](int32_t id) {
        bool part = takes && nparts > 0 && !dead;
        if (WIDE && id < (int32_t)tv.n) {
            const T r2 = ST == ST_GATHER ? ra2 : ex_r2<ST, T>(ra2, __ldg(&tv.nscale[id - 1]), Kt);
            part = part && !(ex_d2_pbox<T>(p, tv, id - 1) > r2);
        } else if (id < (int32_t)tv.n) {
            const float4 lo = __ldg(&tv.node_lo[id - 1]), hi = __ldg(&tv.node_hi[id - 1]);
            part = part && !(lb_d2_pbox(pf, pem, lo, hi) > hi_r2_node<ST>(ra2_hi, lo.w, tv.Kf));
        }
        const unsigned parts = __ballot_sync(PSB_FULL, part);
        if (!parts) {
            ++misses;
            return;
        }
        int64_t lo;
        int cnt;
        span_of(id, lo, cnt);
        if constexpr (WIDE) {
            emit(lo, wide_leaves(lo, cnt, parts, std::integral_constant<int, ST>()));
            ++n_spans;
            n_parts += __popc(parts);
            return;
        }
        // few samples take part: lane j tests leaf j against each of them;
        // otherwise each taking lane tests its sample against every leaf
        const bool by_sample = 3 * __popc(parts) >= 2 * cnt;  // warp-uniform
        // the leaf of this lane with its squared radius (K hb)^2
        float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane < cnt) L = __ldg(&tv.leaf4[lo + lane]);
        float tol = -1.f;  // a pair within it of its squared radius is undecided (double inputs)
        if constexpr (BAND) {
            // one error bound E for every float distance of the span
            float o[3];
            const float2 sb = __ldg(&tv.spanb[lo]);
            const float eqm = anchor(lo, o, sb.x);
            // the rounding of r itself enters through 4 U1 r (r <= the larger radius)
            float rmax = rahimax;
            if (ST != ST_GATHER) rmax = fmaxf(rmax, tv.Kf * sb.y * (1.f + 3.f * U1));
            const float E = 1.7320508f * (esmax + eqm) + 4.f * U1 * rmax + 1e-18f;
            // |d - d_exact| <= E, so d^2 and the exact distance lie on the same side of r^2 unless
            // |d^2 - r^2| <= 2 r E + E^2 (and the roundings of r^2 and of the difference)
            tol = ((2.f * rmax + E) * E + 8.f * U1 * rmax * rmax) * (1.f + 1e-3f);
            L.x += o[0]; L.y += o[1]; L.z += o[2];
            const float kb = tv.Kf * L.w;
            L.w = kb * kb;
        } else if (ST != ST_GATHER) {
            // (no pair is within a radius of NaN: staged as one that nothing is within)
            L.w = fmaxf(ex_r2<ST_SCATTER, float>(0.f, L.w, (float)Kt), -1.f);
        }
        const float Ts = (float)ra2;  // the sample's squared radius
        unsigned myacc = 0;
        float near = INFINITY;  // smallest |d^2 - r^2| of this lane's tests
        __syncwarp();
        if (by_sample) {
            st.put(lane, cnt, L.x, L.y, L.z, L.w);
            __syncwarp();
            if (part) {
                const float4 P = st.P[lane];
                const uint64_t px = pk(P.x, P.x), py = pk(P.y, P.y), pz = pk(P.z, P.z);
                unsigned m = 0;
#pragma unroll 2
                for (int j = (cnt - 1) >> 1; j >= 0; --j) {
                    const LeafPair q = st.L[j];
                    const float2 d2 = pair_d2<!BAND>(px, py, pz, q);
                    float T0 = Ts, T1 = Ts;
                    if (ST == ST_SCATTER) { T0 = q.T.x; T1 = q.T.y; }
                    if (ST == ST_SYMMETRIC) { T0 = fmaxf(Ts, q.T.x); T1 = fmaxf(Ts, q.T.y); }
                    if constexpr (BAND) {  // inside: d^2 - r^2 < 0
                        const float t0 = d2.x - T0, t1 = d2.y - T1;
                        m = push_sign(push_sign(m, t1), t0);
                        near = fminf(near, fminf(fabsf(t0), fabsf(t1)));
                    } else {               // outside: r^2 - d^2 < 0
                        m = push_sign(push_sign(m, T1 - d2.y), T0 - d2.x);
                    }
                }
                myacc = (BAND ? m : ~m) & (0xffffffffu >> (32 - cnt));
            }
        } else {
            st.P[lane].w = Ts;
            __syncwarp();
            for (unsigned pp = parts; pp; pp &= pp - 1) {
                const int s = __ffs(pp) - 1;
                const float4 P = st.P[s];
                const float dx = P.x - L.x, dy = P.y - L.y, dz = P.z - L.z;
                const float Tp = (ST == ST_GATHER) ? P.w : ((ST == ST_SCATTER) ? L.w : fmaxf(P.w, L.w));
                bool in;
                if constexpr (BAND) {
                    const float t = dx * dx + dy * dy + dz * dz - Tp;
                    in = t < 0.f;
                    if (lane < cnt) near = fminf(near, fabsf(t));
                } else {
                    in = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)) <= Tp;
                }
                const unsigned b = __ballot_sync(PSB_FULL, lane < cnt && in);
                if (lane == s) myacc = b;
            }
        }
        if (BAND && __any_sync(PSB_FULL, near <= tol)) {
            // an undecided pair: the reference's double test for the span's (rare)
            if (part) {
                n_retest += cnt;
                myacc = 0;
                for (int j = 0; j < cnt; ++j) {
                    const int64_t li = lo + j;
                    const T e2 = ex_d2_pp<T>(p, __ldg(&tv.x[li]), __ldg(&tv.y[li]), __ldg(&tv.z[li]));
                    myacc |= (unsigned)(e2 <= ex_r2<ST, T>(ra2, __ldg(&tv.h[li]), Kt)) << j;
                }
            }
        }
        emit(lo, myacc);
        ++n_spans;
        n_parts += __popc(parts);
    };
    ok = window_walk<true>(tv, st.q, node_ok, span_fn, steps) && ok;

    const int n0 = chunk >= 0 ? RCAP : nent;  // entries in the tile's list
    if (mine) {
        if (chunk >= 0) {
            A.sp.ccnt[chunk] = (uint8_t)nent;
            A.sp.next[chunk] = -1;
        } else {
            A.sp.head[slot] = -1;
        }
        A.sp.cnt[slot] = dead ? CNT_DEAD : (nparts == 0 ? CNT_HEAVY : (uint8_t)n0);
        ((T*)A.sp.ha)[slot] = ha;
    }
    if (BAND && A.sp.eshift && !dead && nparts > 0 && n0 > 0) {
        // the column shifts of this lane's entries, A[lo] - A0 (span_shift),
        // after the walk: here the entries' loads are independent and overlap,
        // where inside the walk each would stall it.  A0 are the column values
        // of the first accepted leaf.
        const int kc = A.rec.kc;
        const size_t q0 = (size_t)bt * RCAP * 32 + (slot & 31);
        const float4* ent4 = A.sp.ent4 + q0;
        float* esh = A.sp.eshift + (size_t)bt * RCAP * kc * 32 + (slot & 31);
        const int32_t fl = __float_as_int(ent4[0].w) + __ffs(A.sp.emask[q0]) - 1;
        for (int c = 0; c < kc; ++c) {
#pragma unroll 4
            for (int e = 0; e < n0; ++e)
                esh[((size_t)e * kc + c) * 32] = span_shift(A.colT[c], (int64_t)__float_as_int(ent4[(size_t)e * 32].w), fl);
        }
        for (int32_t q = chunk >= 0 ? A.sp.head[slot] : -1; q >= 0; q = A.sp.next[q]) {
            const size_t e0 = (size_t)A.sp.ebase + (size_t)q * RCAP;
            const int n = A.sp.ccnt[q];
            for (int c = 0; c < kc; ++c)
                for (int e = 0; e < n; ++e)
                    A.sp.eshift[(e0 + e) * kc + c] = span_shift(A.colT[c], (int64_t)__float_as_int(A.sp.ent4[e0 + e].w), fl);
        }
    }
    if (valid && A.ha_out) A.ha_out[k] = ha;
    if (dead && lane == 0) list_dead(A.sp, (uint32_t)bt, 0xffffffffu >> (32 - (1 << lspt)) << s0);
    // the single-kernel pass counts the pairs of dead samples, k_heavy those of its samples
    unsigned long long t_pairs = (dead || nparts == 0) ? 0ull : n_pairs, t_retest = n_retest;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t_pairs += __shfl_xor_sync(PSB_FULL, t_pairs, o);
        t_retest += __shfl_xor_sync(PSB_FULL, t_retest, o);
    }
    if (lane == 0 && A.stats) {
        atomicAdd(&A.stats[0], t_pairs);
        atomicAdd(&A.stats[1], t_retest);
        atomicAdd(&A.stats[2], (unsigned long long)steps);
        atomicAdd(&A.stats[3], (unsigned long long)n_spans);
        atomicAdd(&A.stats[4], (unsigned long long)n_parts);
    }
    if (!ok && lane == 0) atomicOr(A.err, PSB_DERR_TRAVERSAL);
}

// The pair lists of the samples whose neighbourhoods outgrew their tile's walk
// (HEAVY_PARTS parts): one CTA per sample.  The walk is a frontier of tree
// nodes in shared memory, expanded level by level in depth-first order (a
// block scan places each node's children where the node was), so that its
// spans end up in leaf order without a serial chain over thousands of nodes;
// then a warp per span tests the leaves with the exact arithmetic, and a scan
// of the non-empty spans gives each entry its place in consecutive chunks.
// The entries are those of the tile's walk, in the same order.  One warp
// walking such a sample alone ran for milliseconds after every other warp had
// finished (150k clump particles, M5, 50k points: 8.0 of 13.5 ms).
constexpr int HEAVY_THREADS = 512;
constexpr int HEAVY_CAP = 12288;  // frontier nodes (a sample of more goes to k_points)
constexpr size_t HEAVY_SMEM = 2 * HEAVY_CAP * sizeof(int32_t);
constexpr int HEAVY_IPT = HEAVY_CAP / HEAVY_THREADS;  // items of a thread
static_assert(HEAVY_IPT <= 32, "two bits per item in a 64-bit word");

// exclusive scan of one value per thread; *total = the sum (all threads call)
static __device__ __forceinline__ int heavy_scan(int v, int* wt, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(PSB_FULL, s, o);
        if (lane >= o) s += t;
    }
    __syncthreads();  // the last scan's totals are read
    if (lane == 31) wt[w] = s;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int q = 0; q < HEAVY_THREADS / 32; ++q) {
        const int t = wt[q];
        if (q < w) before += t;
        all += t;
    }
    *total = all;
    return before + s - v;
}

template <class T, int ST>
__global__ void __launch_bounds__(HEAVY_THREADS, 2) k_heavy(const Args<T> A) {
    extern __shared__ __align__(16) int32_t hbuf[];
    __shared__ int wt[HEAVY_THREADS / 32];
    // two words: a warp may still read one sample's s_base when thread 0 is at the next sample's s_skip
    __shared__ unsigned s_skip, s_base;
    const TreeView<T>& tv = A.tv;
    const SplitBufs& sp = A.sp;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned nh = min(*sp.hcount, sp.hcap);
    for (unsigned i = blockIdx.x; i < nh; i += gridDim.x) {
        const uint32_t idx = sp.hlist[i];
        // a sample whose warp found the pool empty is k_points' already; with
        // the pool empty no other sample is worth its walk
        if (tid == 0) s_skip = sp.cnt[idx] == CNT_DEAD ? 2u : (atomicAdd(sp.top, 0u) >= sp.ncap ? 1u : 0u);
        __syncthreads();
        const unsigned give_up = s_skip;
        __syncthreads();
        if (give_up) {
            if (give_up == 1u && tid == 0) {
                sp.cnt[idx] = CNT_DEAD;
                list_dead(sp, idx >> 5, 1u << (idx & 31));
            }
            continue;
        }
        const int64_t k = sample_of(A.src, sp.tile0 + (idx >> 5), idx & 31);
        T p[3], dd[3];
        sample_coords(A.src, k, p, dd);
        const T ha = ((const T*)sp.ha)[idx];
        const float pf[3] = {(float)p[0], (float)p[1], (float)p[2]};
        const float pem = U1 * fmaxf(fmaxf(fabsf(pf[0]), fabsf(pf[1])), fabsf(pf[2])) + 1e-30f;
        const T Kt = (T)tv.Kd;
        const T ra = X<T>::mul(Kt, ha);
        const T ra2 = X<T>::mul(ra, ra);
        const float ra2_hi = (ST == ST_SCATTER) ? 0.f : __double2float_ru((double)ra2) * (1.f + RELM) + 1e-36f;
        int32_t* cur = hbuf;
        int32_t* nxt = hbuf + HEAVY_CAP;
        // items: a node still to be tested (id > 0) or a span (-id); the root
        // has more than SPAN leaves (its sample has more than one span)
        __syncthreads();
        if (tid == 0) cur[0] = tv.root;
        __syncthreads();
        int f = 1;
        bool fits = true;
        for (int level = 0;; ++level) {
            const int ipt = (f + HEAVY_THREADS - 1) / HEAVY_THREADS;
            const int a = min(f, tid * ipt), b = min(f, a + ipt);
            unsigned long long res = 0;  // per item: 0 none, 1 a span, 2 its two children
            int out = 0;
            bool open = false;
            for (int q = a; q < b; ++q) {
                const int32_t id = cur[q];
                unsigned r = 1;
                if (id > 0 && id < tv.n) {
                    const int4 lk = __ldg(&tv.links[id - 1]);
                    const float4 lo = __ldg(&tv.node_lo[id - 1]), hi = __ldg(&tv.node_hi[id - 1]);
                    if (lb_d2_pbox(pf, pem, lo, hi) > hi_r2_node<ST>(ra2_hi, lo.w, tv.Kf)) r = 0;
                    else if (lk.w - lk.z + 1 > SPAN) { r = 2; open = true; }
                }
                res |= (unsigned long long)r << (2 * (q - a));
                out += (int)r;
            }
            int nf;
            int w = heavy_scan(out, wt, &nf);
            if (nf > HEAVY_CAP || level > 4 * 64) { fits = false; break; }  // (a corrupt tree never closes)
            for (int q = a; q < b; ++q) {
                const int32_t id = cur[q];
                const unsigned r = (unsigned)(res >> (2 * (q - a))) & 3u;
                if (r == 1) {
                    nxt[w++] = id > 0 ? -id : id;
                } else if (r == 2) {
                    nxt[w++] = __ldg(&tv.left[id - 1]);
                    nxt[w++] = __ldg(&tv.right[id - 1]);
                }
            }
            open = __syncthreads_or(open);
            int32_t* t = cur; cur = nxt; nxt = t;
            f = nf;
            if (!open) break;
        }
        if (fits) {
            // accept masks of the spans (nxt), a warp per span
            uint32_t* msk = (uint32_t*)nxt;
            unsigned n_pairs = 0;
#pragma unroll 2
            for (int q = warp; q < f; q += HEAVY_THREADS / 32) {
                const int32_t id = -cur[q];
                int64_t lo;
                int cnt;
                if (id >= tv.n) {
                    lo = (int64_t)id - tv.n;
                    cnt = 1;
                } else {
                    const int4 lk = __ldg(&tv.links[id - 1]);
                    lo = (int64_t)lk.z - 1;
                    cnt = lk.w - lk.z + 1;
                }
                bool in = false;
                if (lane < cnt) {
                    const int64_t li = lo + lane;
                    const T e2 = ex_d2_pp<T>(p, __ldg(&tv.x[li]), __ldg(&tv.y[li]), __ldg(&tv.z[li]));
                    in = e2 <= ex_r2<ST, T>(ra2, __ldg(&tv.h[li]), Kt);
                }
                const unsigned m = __ballot_sync(PSB_FULL, in);
                __syncwarp();
                if (lane == 0) {
                    cur[q] = (int32_t)lo;  // the entry's first leaf
                    msk[q] = m;
                }
                n_pairs += __popc(m);
            }
            __syncthreads();
            const int ipt = (f + HEAVY_THREADS - 1) / HEAVY_THREADS;
            const int a = min(f, tid * ipt), b = min(f, a + ipt);
            int out = 0;
            for (int q = a; q < b; ++q) out += msk[q] != 0;
            int ne;
            int w = heavy_scan(out, wt, &ne);
            const unsigned nch = (unsigned)((ne + RCAP - 1) / RCAP);
            if (tid == 0) s_base = atomicAdd(sp.top, nch);
            __syncthreads();
            const unsigned base = s_base;
            fits = base < sp.ncap && nch <= sp.ncap - base;
            for (unsigned c = tid; c < nch; c += HEAVY_THREADS) {
                if (base + c >= sp.ncap) break;
                sp.own[base + c] = fits ? (idx | OWN_HEAVY | (c ? OWN_LATER : 0u)) : OWN_NONE;
                sp.next[base + c] = c + 1 < nch ? (int32_t)(base + c + 1) : -1;
                sp.ccnt[base + c] = (uint8_t)min(RCAP, ne - (int)c * RCAP);
            }
            if (fits) {
                const size_t e0 = (size_t)sp.ebase + (size_t)base * RCAP;
                const size_t q0 = (size_t)(idx >> 5) * RCAP * 32 + (idx & 31);
                // A0 of the column shifts: the sample's first accepted leaf (its list's first pair)
                const int32_t fl = __float_as_int(sp.ent4[q0].w) + __ffs(sp.emask[q0]) - 1;
                for (int q = a; q < b; ++q) {
                    if (!msk[q]) continue;
                    const int64_t lo = cur[q];
                    float r0 = 0.f, r1 = 0.f, r2 = 0.f;
                    if (sizeof(T) == 8 && !sp.fp64) {
                        r0 = (float)((double)p[0] - (double)__ldg(&tv.x[lo]));
                        r1 = (float)((double)p[1] - (double)__ldg(&tv.y[lo]));
                        r2 = (float)((double)p[2] - (double)__ldg(&tv.z[lo]));
                    }
                    sp.ent4[e0 + w] = make_float4(r0, r1, r2, __int_as_float((int)lo));
                    sp.emask[e0 + w] = msk[q];
                    if (sp.eshift)
                        for (int c = 0; c < A.rec.kc; ++c)
                            sp.eshift[(e0 + w) * A.rec.kc + c] = span_shift(A.colT[c], lo, fl);
                    ++w;
                }
                if (A.stats && lane == 0) atomicAdd(&A.stats[0], (unsigned long long)n_pairs);
                if (A.stats && tid == 0) {
                    atomicAdd(&A.stats[3], (unsigned long long)f);
                    atomicAdd(&A.stats[4], (unsigned long long)f);
                }
                if (sp.mlist && tid == 0) sp.mlist[atomicAdd(sp.mcount, 1u)] = base;
            }
        }
        if (!fits && tid == 0) {  // k_points takes the sample
            sp.cnt[idx] = CNT_DEAD;
            list_dead(sp, idx >> 5, 1u << (idx & 31));
        }
    }
}

// The data of one pair for k_bodies: the double records for the FP64 sums, the
// float records for FP32C (with double inputs relative to the span's first leaf).
template <class T, int PREC, int KC> struct PairData {  // PREC_FP64
    double2 a, b, s;  // (x, y), (z, 1/h), (sigma/h^3, m/rho)
    T mb;             // mass (density gradient only)
    T col[KC];
    __device__ __forceinline__ void load(const TreeView<T>& tv, const Args<T>& A, int64_t li, int kc, bool need_dg,
                                         const float*, const float* const*) {
        a = __ldg(&tv.leafD[0][li]); b = __ldg(&tv.leafD[1][li]); s = __ldg(&tv.leafD[2][li]);
        mb = need_dg ? __ldg(&tv.m[li]) : T(0);
#pragma unroll
        for (int c = 0; c < KC; ++c) col[c] = (c < kc) ? __ldg(&A.colT[c][li]) : T(0);
    }
};
template <int KC> struct PairData<float, PREC_FP32C, KC> {
    float4 L, K;  // leaf4 (the exact position and h) and leafK
    float mb;
    float col[KC];
    __device__ __forceinline__ void load(const TreeView<float>& tv, const Args<float>& A, int64_t li, int kc,
                                         bool need_dg, const float*, const float* const*) {
        L = __ldg(&tv.leaf4[li]);
        K = __ldg(&tv.leafK[li]);
        mb = need_dg ? __ldg(&tv.m[li]) : 0.f;
#pragma unroll
        for (int c = 0; c < KC; ++c) col[c] = (c < kc) ? __ldg(&A.colT[c][li]) : 0.f;
    }
};
template <int KC> struct PairData<double, PREC_FP32C, KC> {
    using T = double;
    float4 L, K;      // leaf4 and leafK of the particle
    float col[KC];    // the column in float, or for EXS span-relative (A - A0 once the entry's shift is added)
    float mb;         // mass (density gradient only)
    float r[3];       // the sample relative to the span's first leaf
    int64_t li;       // leaf index
    double xd, yd, zd, hd;  // the particle in double (outer kernel piece)
    __device__ __forceinline__ void load(const TreeView<T>& tv, const Args<T>& A, int64_t li, int kc, bool need_dg,
                                         const float* Rs, const float* const* cols) {
        L = __ldg(&tv.leaf4[li]);
        K = __ldg(&tv.leafK[li]);
#pragma unroll
        for (int c = 0; c < KC; ++c) col[c] = (c < kc) ? __ldg(&cols[c][li]) : 0.f;
        mb = need_dg ? __ldg(&tv.mf[li]) : 0.f;
        r[0] = Rs[0]; r[1] = Rs[1]; r[2] = Rs[2];
        this->li = li;
        xd = __ldg(&tv.x[li]); yd = __ldg(&tv.y[li]); zd = __ldg(&tv.z[li]); hd = __ldg(&tv.h[li]);
    }
};

// FP32C of double particles, samples of several parts: from CHAIN_SAMPLES of them
// in a batch on, those of few parts go to k_bodies and k_density with a lane per
// sample (CHAIN), the others stay k_seq's, whose warp takes a sample in order at
// a third of the rate but does not wait for the longest of 32.  729,000 grid points,
// gather, FP32C: 1000 particles of a Plummer sphere 9.0 -> 6.6 ms (M6 18.1 -> 10.9),
// 20,000 of clumps 8.4 -> 8.4 (M6 29 -> 30); from 16,384 samples on 6.0 and 7.5, but
// 200,000 points about 300,000 clump particles 5.4 -> 6.7.
constexpr unsigned CHAIN_SAMPLES = 65536;
// whether a sample (its first chunk and that chunk's owner word) has more than HEAVY_PARTS parts
__device__ __forceinline__ bool long_chain(const SplitBufs& sp, int32_t c, uint32_t own) {
    if (own & OWN_HEAVY) return true;
    int parts = 1;  // the tile's list
    for (; c >= 0 && parts <= HEAVY_PARTS; c = sp.next[c]) ++parts;
    return parts > HEAVY_PARTS;
}

// The list part of a thread of the pair-sum kernels.  Blocks below `nlist` take
// some tiles' lists (a warp per tile, one lane per sample), the blocks after
// them a chunk of the pool per thread.
struct ListPart {
    int64_t bt;      // the sample's tile in the batch
    int lane;        // and its lane there
    int n;           // entries (0: nothing to do)
    uint32_t e0;     // index of the first entry
    int step;        // distance of consecutive entries
    int32_t chunk;   // the chunk, or -1 for a list
    int32_t dst;     // chunk whose partial sums this part writes, or -1: the sample's only part
};
__device__ __forceinline__ ListPart list_part(const SplitBufs& sp, unsigned nlist) {
    ListPart q;
    q.n = 0;
    q.dst = -1;
    q.lane = threadIdx.x & 31;
    if (blockIdx.x < nlist) {
        q.bt = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
        q.chunk = -1;
        q.e0 = (uint32_t)q.bt * (RCAP * 32) + q.lane;
        q.step = 32;
        if (q.bt < sp.ntiles) {
            const int n = sp.cnt[q.bt * 32 + q.lane];
            q.n = n >= CNT_HEAVY ? -1 : n;  // -1: the single-kernel pass's tile, or k_heavy's sample
            q.dst = n == RCAP ? sp.head[q.bt * 32 + q.lane] : -1;
            if (sp.mlist && q.dst >= 0) q.n = -1;  // k_seq's
        } else {
            q.n = -1;
        }
        return q;
    }
    const unsigned c = (blockIdx.x - nlist) * blockDim.x + threadIdx.x;
    const unsigned used = min(*sp.top, sp.ncap);
    q.bt = 0;
    q.chunk = (int32_t)c;
    q.e0 = sp.ebase + c * RCAP;
    q.step = 1;
    q.n = -1;
    if (c < used) {
        const uint32_t w = sp.own[c], o = w & OWN_IDX;
        if (w != OWN_NONE) {
            q.bt = o >> 5;
            q.lane = (int)(o & 31);
            const int n = sp.cnt[o];
            // a sample handed to k_heavy leaves the chunks of its tile's walk behind
            if (n != CNT_DEAD && (n == CNT_HEAVY) == ((w & OWN_HEAVY) != 0)) {
                q.n = sp.ccnt[c];
                q.dst = (int32_t)c;
            }
        }
    }
    return q;
}

// The same for sums that run on through a sample's parts with a lane per sample
// (CHAIN): a thread takes a sample of up to HEAVY_PARTS parts, from its first on.
__device__ __forceinline__ ListPart chain_part(const SplitBufs& sp) {
    ListPart q;
    q.n = -1;
    q.dst = -1;
    q.bt = 0;
    q.lane = threadIdx.x & 31;
    q.chunk = -1;
    q.e0 = 0;
    q.step = 32;
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x, count = min(*sp.mcount, sp.ncap);
    if (i >= count || count < CHAIN_SAMPLES) return q;
    const int32_t c = (int32_t)sp.mlist[i];
    const uint32_t w = sp.own[c], o = w & OWN_IDX;
    if (sp.cnt[o] >= CNT_HEAVY || long_chain(sp, c, w)) return q;  // k_seq's, or the single kernel's
    q.bt = o >> 5;
    q.lane = (int)(o & 31);
    q.e0 = (uint32_t)q.bt * (RCAP * 32) + q.lane;
    q.n = RCAP;
    return q;
}

template <class T, int PREC, int ST, int KC, int KF, bool DG, bool CHAIN = false>
__global__ void __launch_bounds__(BODY_THREADS, 128 / BODY_THREADS * ((KC <= 4 || (KC == 5 && sizeof(T) == 4)) ? 4 : (KC <= 6 ? 3 : 2)))
    k_bodies(const Args<T> A, unsigned nlist) {
    using CT = typename std::conditional<PREC == PREC_FP64, double, float>::type;
    using Acc = typename std::conditional<PREC == PREC_FP64, PlainD, KahanF>::type;
    constexpr bool BAND = (PREC == PREC_FP32C) && (sizeof(T) == 8);
    constexpr bool SHIFT = (PREC == PREC_FP32C);
    constexpr bool EXS = BAND && KF == 1;  // column shifts formed in double (span_shift), from k_collect
    const TreeView<T>& tv = A.tv;
    const ListPart Q = CHAIN ? chain_part(A.sp) : list_part(A.sp, nlist);
    if (!__any_sync(PSB_FULL, Q.n >= 0)) return;
    int n = max(Q.n, 0);
    const int64_t bt = Q.bt;
    const int lane = Q.lane;  // the sample's lane in its tile
    const int64_t tile = A.sp.tile0 + bt;
    const int64_t k = Q.n >= 0 ? sample_of(A.src, tile, lane) : -1;
    const bool valid = k >= 0;
    T p[3] = {T(0), T(0), T(0)}, dd[3];
    if (valid) sample_coords(A.src, k, p, dd);
    const T ha = ((const T*)A.sp.ha)[bt * 32 + lane];
    const int kc = A.rec.kc;
    constexpr bool need_dg = DG;  // A.rec.need_dg (the launch picks the instantiation)

    const CT sig = (KF == 0) ? inv_pi<CT>() : (CT)tv.sig;
    CT ia = CT(0), sa3 = CT(0), sa4 = CT(0);
    if (ST != ST_SCATTER) {
        ia = CT(1) / (CT)ha;
        sa3 = sig * ia * ia * ia;
        sa4 = sa3 * ia;
    }
    const double kha = tv.Kd * (double)ha;
    const double fa2 = kha * kha;  // (K ha)^2 for the kernel piece at the support edge
    const double ika = (KF == 1 && ST != ST_SCATTER) ? 0.5 / (double)ha : 0.0;  // Wendland pair terms
    const float qe = (KF == 0) ? 1.f : tv.qedge;
    Acc S1, G[3], Sw[KC], Sg[KC][3], Dm, Dg[3];
    // FP32C sums are of A - A0, A0 the column values of the sample's first
    // accepted leaf (the first pair of its list)
    CT a0[KC];
    int64_t first = -1;
    if (SHIFT && n > 0) {
        const size_t q0 = (size_t)bt * RCAP * 32 + lane;
        first = (int64_t)__float_as_int(A.sp.ent4[q0].w) + __ffs(A.sp.emask[q0]) - 1;
    }
    S1.zero(); Dm.zero();
#pragma unroll
    for (int d = 0; d < 3; ++d) { G[d].zero(); Dg[d].zero(); }
#pragma unroll
    for (int c = 0; c < KC; ++c) {
        Sw[c].zero();
        a0[c] = CT(0);
        if (SHIFT && !EXS && first >= 0 && c < kc) a0[c] = (CT)__ldg(&A.colF[c][first]);
#pragma unroll
        for (int d = 0; d < 3; ++d) Sg[c][d].zero();
    }

    // Kernel weights and sums of one pair; weights as in k_points, every
    // rounding spelled out (acc_mul, acc_mac).
    auto accumulate = [&](const auto& col, CT dx, CT dy, CT dz, CT Wsum, CT csum, CT mr, CT mb) {
        const CT w = acc_mul(mr, Wsum);
        const CT gc = acc_mul(mr, csum);
        const CT gx = acc_mul(gc, dx), gy = acc_mul(gc, dy), gz = acc_mul(gc, dz);
        S1.add(w);
        G[0].add(gx); G[1].add(gy); G[2].add(gz);
#pragma unroll
        for (int c = 0; c < KC; ++c) {
            if (c < kc) {
                CT a = (CT)col[c];  // EXS: already A - A0
                if constexpr (SHIFT && !EXS) a = __fsub_rn(a, a0[c]);
                acc_mac(Sw[c], a, w);
                acc_mac(Sg[c][0], a, gx); acc_mac(Sg[c][1], a, gy); acc_mac(Sg[c][2], a, gz);
            }
        }
        if (need_dg) {
            acc_mac(Dm, mb, Wsum);
            const CT mc = acc_mul(mb, csum);
            acc_mac(Dg[0], mc, dx); acc_mac(Dg[1], mc, dy); acc_mac(Dg[2], mc, dz);
        }
    };

    // The pairs of this lane's list, one ahead: the loads of the next pair are
    // in flight while the current pair is summed.
    const float4* ent4 = A.sp.ent4 + Q.e0;
    const uint32_t* emask = A.sp.emask + Q.e0;
    const float* esh = !EXS ? nullptr
                       : Q.chunk < 0 ? A.sp.eshift + (size_t)bt * RCAP * kc * 32 + lane
                                     : A.sp.eshift + (size_t)Q.e0 * kc;
    int est = Q.step;
    int32_t more = CHAIN && n > 0 ? A.sp.head[bt * 32 + lane] : -1;  // CHAIN: the part after this one
    int e = 0;
    unsigned m = 0;
    int64_t lo = 0;
    float Rs[3] = {0.f, 0.f, 0.f};
    float sh[KC];          // EXS: the entry's column shifts A[lo] - A0 (written by k_collect)
#pragma unroll
    for (int c = 0; c < KC; ++c) sh[c] = 0.f;
    PairData<T, PREC, KC> nx;
    bool hn = false;
    auto fetch = [&]() {
        if (CHAIN && m == 0 && e == n && more >= 0) {
            const size_t e0 = (size_t)A.sp.ebase + (size_t)more * RCAP;
            ent4 = A.sp.ent4 + e0;
            emask = A.sp.emask + e0;
            if (EXS) esh = A.sp.eshift + e0 * kc;
            est = 1;
            e = 0;
            n = A.sp.ccnt[more];
            more = A.sp.next[more];
        }
        if (m == 0 && e < n) {
            const float4 q = ent4[e * est];
            m = emask[e * est];  // never 0: k_collect writes entries with accepted leaves only
            ++e;
            lo = (int64_t)__float_as_int(q.w);
            Rs[0] = q.x; Rs[1] = q.y; Rs[2] = q.z;
            if constexpr (EXS) {
#pragma unroll
                for (int c = 0; c < KC; ++c) sh[c] = (c < kc) ? esh[((e - 1) * kc + c) * est] : 0.f;
            }
        }
        hn = m != 0;
        if (hn) {
            const int j = __ffs(m) - 1;
            m &= m - 1;
            nx.load(tv, A, lo + j, kc, need_dg, Rs, EXS ? A.colR : A.colF);
        }
    };
    unsigned long long n_bodyit = 0;
    fetch();
    while (__any_sync(PSB_FULL, hn)) {
        const bool hc = hn;
        PairData<T, PREC, KC> cur = nx;
        if constexpr (EXS) {
            // A - A0: the shifts of cur's entry (fetch may start the next one);
            // added here, an iteration after the loads, not as they return
#pragma unroll
            for (int c = 0; c < KC; ++c) cur.col[c] = __fadd_rn(cur.col[c], sh[c]);
        }
        fetch();
        ++n_bodyit;
        if (!hc) continue;
        if constexpr (BAND) {
            const float dx = __fsub_rn(cur.r[0], cur.L.x);
            const float dy = __fsub_rn(cur.r[1], cur.L.y);
            const float dz = __fsub_rn(cur.r[2], cur.L.z);
            float Wsum, csum;
            f32c_pair_weights<ST, KF>(
                tv.kern, tv.Kf, qe, dx, dy, dz, (float)ia, (float)sa3, (float)sa4, fa2, ika, (float)ha, cur.K, cur.L.w,
                [&]() {
                    const double ex = __dsub_rn((double)p[0], cur.xd);
                    const double ey = __dsub_rn((double)p[1], cur.yd);
                    const double ez = __dsub_rn((double)p[2], cur.zd);
                    return __fma_rn(ex, ex, __fma_rn(ey, ey, __dmul_rn(ez, ez)));
                },
                [&]() { return __dmul_rn(tv.Kd, cur.hd); }, Wsum, csum);
            accumulate(cur.col, dx, dy, dz, Wsum, csum, cur.K.w, cur.mb);
        } else if constexpr (PREC == PREC_FP64) {
            const double dx = __dsub_rn((double)p[0], cur.a.x), dy = __dsub_rn((double)p[1], cur.a.y),
                         dz = __dsub_rn((double)p[2], cur.b.x);
            double W, cg;
            f64_pair_weights<ST, KF>(tv.kern, dx, dy, dz, ia, sa3, cur.b.y, cur.s.x, W, cg);
            CT cc[KC];
#pragma unroll
            for (int c = 0; c < KC; ++c) cc[c] = (CT)cur.col[c];
            accumulate(cc, dx, dy, dz, W, cg, cur.s.y, (CT)cur.mb);
        } else {
            float W, cg;
            const float dx = __fsub_rn(p[0], cur.L.x), dy = __fsub_rn(p[1], cur.L.y), dz = __fsub_rn(p[2], cur.L.z);
            f32_pair_weights<ST, KF>(tv.kern, ex_d2_pp<T>(p, cur.L.x, cur.L.y, cur.L.z), ia, sa3, sa4, cur.K.x,
                                     cur.K.y, W, cg);
            accumulate(cur.col, dx, dy, dz, W, cg, cur.K.w, cur.mb);
        }
    }

    if (valid && Q.dst >= 0) {
        // one of several parts: its sums, folded by k_fold
        double* o = A.sp.part + (Q.chunk < 0 ? A.sp.ncap : 0) + Q.dst;
        const size_t fs = 2 * (size_t)A.sp.ncap;  // distance of fields
        o[0] = S1.get();
#pragma unroll
        for (int d = 0; d < 3; ++d) o[(1 + d) * fs] = G[d].get();
        if (DG) {
            o[4 * fs] = Dm.get();
#pragma unroll
            for (int d = 0; d < 3; ++d) o[(5 + d) * fs] = Dg[d].get();
        }
#pragma unroll
        for (int c = 0; c < KC; ++c) {
            o[(8 + c) * fs] = Sw[c].get();
#pragma unroll
            for (int d = 0; d < 3; ++d) o[(8 + KC + 3 * c + d) * fs] = Sg[c][d].get();
        }
    } else if (valid) {
        double a0o[KC];
#pragma unroll
        for (int c = 0; c < KC; ++c)
            a0o[c] = EXS ? ((c < kc && first >= 0) ? (double)A.colT[c][first] : 0.0) : (double)a0[c];
        write_interp_outputs<T, Acc, CT, KC>(A, k, S1, G, Sw, Sg, Dm, Dg, a0o);
    }
    if ((threadIdx.x & 31) == 0 && A.stats) atomicAdd(&A.stats[5], n_bodyit);
}

// The density sums over the pair lists (psb_density: sum m W, or sum W with
// unit masses), one lane per sample as in k_bodies, with the arithmetic and
// order of k_points' density.  One sum and no gradient fit 64 registers, so
// the pair loads are hidden by 8 CTAs per SM; the single kernel summed span
// by span behind its walk with a third of its lanes busy
// (1M clump particles, gather at the particles: 10.4 ms in k_points; now the
// walk, k_heavy and this kernel take 3.5 ms).
template <class T, int PREC, int ST, int KF, bool CHAIN = false>
__global__ void __launch_bounds__(BODY_THREADS, 1024 / BODY_THREADS) k_density(const Args<T> A, unsigned nlist) {
    using CT = typename std::conditional<PREC == PREC_FP64, double, float>::type;
    using Acc = typename std::conditional<PREC == PREC_FP64, PlainD, KahanF>::type;
    constexpr bool BAND = (PREC == PREC_FP32C) && (sizeof(T) == 8);
    const TreeView<T>& tv = A.tv;
    const ListPart Q = CHAIN ? chain_part(A.sp) : list_part(A.sp, nlist);
    int n = Q.n;
    const int64_t k = n < 0 ? -1 : sample_of(A.src, A.sp.tile0 + Q.bt, Q.lane);
    const unsigned active = __ballot_sync(PSB_FULL, k >= 0);
    if (k < 0) return;
    T p[3], dd[3];
    sample_coords(A.src, k, p, dd);
    const T ha = ((const T*)A.sp.ha)[Q.bt * 32 + Q.lane];
    const CT sig = (KF == 0) ? inv_pi<CT>() : (CT)tv.sig;
    CT ia = CT(0), sa3 = CT(0), sa4 = CT(0);
    if (ST != ST_SCATTER) {
        ia = CT(1) / (CT)ha;
        sa3 = sig * ia * ia * ia;
        sa4 = sa3 * ia;
    }
    const double kha = tv.Kd * (double)ha;
    const double fa2 = kha * kha;
    const double ika = (KF == 1 && ST != ST_SCATTER) ? 0.5 / (double)ha : 0.0;
    const float qe = (KF == 0) ? 1.f : tv.qedge;
    const bool unit = A.unit_mass != 0;
    Acc D;
    D.zero();
    const float4* ent4 = A.sp.ent4 + Q.e0;
    const uint32_t* emask = A.sp.emask + Q.e0;
    int est = Q.step;
    int32_t more = CHAIN ? A.sp.head[Q.bt * 32 + Q.lane] : -1;  // CHAIN: the part after this one
    PairData<T, PREC, 1> nx;
    float Rs[3] = {0.f, 0.f, 0.f};
    int e = 0;
    unsigned m = 0;
    int64_t lo = 0;
    auto fetch = [&]() -> bool {
        if (m == 0) {
            if (e >= n) {
                if (!CHAIN || more < 0) return false;
                const size_t e0 = (size_t)A.sp.ebase + (size_t)more * RCAP;
                ent4 = A.sp.ent4 + e0;
                emask = A.sp.emask + e0;
                est = 1;
                e = 0;
                n = A.sp.ccnt[more];
                more = A.sp.next[more];
            }
            const float4 q = ent4[e * est];
            m = emask[e * est];
            ++e;
            lo = (int64_t)__float_as_int(q.w);
            Rs[0] = q.x; Rs[1] = q.y; Rs[2] = q.z;
        }
        const int j = __ffs(m) - 1;
        m &= m - 1;
        nx.load(tv, A, lo + j, 0, !unit, Rs, nullptr);
        return true;
    };
    unsigned n_bodyit = 0;
    bool has = fetch();
    while (has) {
        const PairData<T, PREC, 1> cur = nx;
        has = fetch();
        ++n_bodyit;
        CT W, c;
        if constexpr (BAND) {
            f32c_pair_weights<ST, KF>(
                tv.kern, tv.Kf, qe, __fsub_rn(cur.r[0], cur.L.x), __fsub_rn(cur.r[1], cur.L.y),
                __fsub_rn(cur.r[2], cur.L.z), (float)ia, (float)sa3, (float)sa4, fa2, ika, (float)ha, cur.K, cur.L.w,
                [&]() {
                    const double ex = __dsub_rn((double)p[0], cur.xd);
                    const double ey = __dsub_rn((double)p[1], cur.yd);
                    const double ez = __dsub_rn((double)p[2], cur.zd);
                    return __fma_rn(ex, ex, __fma_rn(ey, ey, __dmul_rn(ez, ez)));
                },
                [&]() { return __dmul_rn(tv.Kd, cur.hd); }, W, c);
        } else if constexpr (PREC == PREC_FP64) {
            f64_pair_weights<ST, KF>(tv.kern, __dsub_rn((double)p[0], cur.a.x), __dsub_rn((double)p[1], cur.a.y),
                                     __dsub_rn((double)p[2], cur.b.x), ia, sa3, cur.b.y, cur.s.x, W, c);
        } else {
            f32_pair_weights<ST, KF>(tv.kern, ex_d2_pp<T>(p, cur.L.x, cur.L.y, cur.L.z), ia, sa3, sa4, cur.K.x,
                                     cur.K.y, W, c);
        }
        acc_mac(D, unit ? CT(1) : (CT)cur.mb, W);
    }
    if (Q.dst >= 0) A.sp.part[(Q.chunk < 0 ? A.sp.ncap : 0) + Q.dst] = D.get();
    else A.out[0][k] = (PREC == PREC_FP64) ? (T)D.get() : (T)(CT)D.get();
    n_bodyit = __reduce_max_sync(active, n_bodyit);
    if (A.stats && (int)(threadIdx.x & 31) == __ffs(active) - 1) atomicAdd(&A.stats[5], (unsigned long long)n_bodyit);
}

// The samples of several list parts: the list's sums, then the chunks' in the
// chain's order, added up; then the outputs (all but FP32C of double
// particles, see k_seq).  One thread per chunk of the pool; a sample's first
// chunk does the work.  WHAT is k_points'.
template <class T, int PREC, int KC, int WHAT>
__global__ void __launch_bounds__(128) k_fold(const Args<T> A) {
    using CT = typename std::conditional<PREC == PREC_FP64, double, float>::type;
    const unsigned c0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (c0 >= min(*A.sp.top, A.sp.ncap)) return;
    const uint32_t w = A.sp.own[c0], own = w & OWN_IDX;
    if (w & OWN_LATER) return;  // a later chunk, or none
    const int cn = A.sp.cnt[own];
    const bool heavy = (w & OWN_HEAVY) != 0;
    if (cn == CNT_DEAD || (cn == CNT_HEAVY) != heavy) return;
    const int64_t k = sample_of(A.src, A.sp.tile0 + (own >> 5), own & 31);
    if (k < 0) return;
    // the first part: the tile's list, or a heavy sample's first chunk
    const size_t f0 = heavy ? c0 : A.sp.ncap + c0;
    const int32_t c1 = heavy ? A.sp.next[c0] : (int32_t)c0;
    const size_t fs = 2 * (size_t)A.sp.ncap;
    if (WHAT == WHAT_DENSITY) {
        double t = A.sp.part[f0];
        for (int32_t c = c1; c >= 0; c = A.sp.next[c]) t = __dadd_rn(t, A.sp.part[c]);
        A.out[0][k] = (PREC == PREC_FP64) ? (T)t : (T)(CT)t;
        return;
    }
    constexpr int NF = 8 + 4 * KC;
    double t[NF];
    const bool dg = A.rec.need_dg != 0;
#pragma unroll
    for (int q = 0; q < NF; ++q) t[q] = (q >= 4 && q < 8 && !dg) ? 0.0 : A.sp.part[q * fs + f0];
    for (int32_t c = c1; c >= 0; c = A.sp.next[c]) {
#pragma unroll
        for (int q = 0; q < NF; ++q)
            if (!(q >= 4 && q < 8) || dg) t[q] = __dadd_rn(t[q], A.sp.part[q * fs + c]);
    }
    PlainD S1, G[3], Dm, Dg[3], Sw[KC], Sg[KC][3];
    S1.s = t[0];
    Dm.s = t[4];
#pragma unroll
    for (int d = 0; d < 3; ++d) { G[d].s = t[1 + d]; Dg[d].s = t[5 + d]; }
    double a0[KC];
    const size_t q0 = (size_t)(own >> 5) * RCAP * 32 + (own & 31);
    const int64_t first = (int64_t)__float_as_int(A.sp.ent4[q0].w) + __ffs(A.sp.emask[q0]) - 1;
#pragma unroll
    for (int c = 0; c < KC; ++c) {
        Sw[c].s = t[8 + c];
#pragma unroll
        for (int d = 0; d < 3; ++d) Sg[c][d].s = t[8 + KC + 3 * c + d];
        a0[c] = (PREC == PREC_FP64 || c >= A.rec.kc) ? 0.0
                : (double)A.colF[c][first];
    }
    write_interp_outputs<T, PlainD, CT, KC>(A, k, S1, G, Sw, Sg, Dm, Dg, a0);
}

// One warp per sample: in FP32C of double particles for the samples of several
// list parts, whose sums run on through the parts, and in small calls for every
// sample (seq_all; parts of FP64 and float particles' samples are summed apart,
// as in k_bodies).  A part's pairs are taken 32 at a time, whatever entries they
// come from: lane j evaluates the weights of pair j, with k_bodies' arithmetic;
// then each sum runs through those pairs in order in a lane of its own (4 + 4 kc
// sums, 4 more with a density gradient, two to a lane past 32).  The sums have
// the bits of one lane adding pair after pair.
//
// Bound by the latency of the records and of the compensated chain (four
// dependent operations a pair).  FP32C of samples of several parts, 4 columns:
// taken entry by entry, with the lanes of an entry's accepted leaves (some 16 of
// 32) at work, 524,288 samples of 1922 neighbours on average (a tenth of them
// have most, up to 45,000) took 82 ms a call, in windows 51; the tiles' walk
// and single kernel that such samples took before there were parts, 53.  M6: 154, 99,
// 92; 500,000 points about clumps (M6) 72, 40, 104.  A lane per sample through
// all its parts, however many: 93 and 163, 90 (see CHAIN_SAMPLES).
//
// A small call is as long as its longest lane: 37 points waited 230 us for
// k_bodies.  1M uniform particles, scatter, 12 FP64 outputs, a call of 32
// points takes 126 us (k_bodies 170), 1024 202 (241), 4096 274 (317), 8192 366
// (390), 16,384 420 (418), 65,536 753 (559); the density alone 123 (159), 194
// (230), 234 (292), 318 (377), 349 (402), 517 (514).  FP32C and float particles
// cross at 8192 to 16,384 points as well; the line stays below that.
constexpr int SEQ_COMP = 8;  // weights of a pair: w, w d (3); with a density gradient W, d (3); then the columns, m, m W'
constexpr int SEQ_ROWS = SEQ_COMP + MAX_KC + 2;
constexpr int64_t SEQ_ALL = 4096;  // samples of a call up to which k_seq takes all
template <class T, int PREC, int ST, int KF, int WHAT>
__global__ void __launch_bounds__(128) k_seq(const __grid_constant__ Args<T> A) {
    using CT = typename std::conditional<PREC == PREC_FP64, double, float>::type;
    using Acc = typename std::conditional<PREC == PREC_FP64, PlainD, KahanF>::type;
    constexpr bool BAND = PREC == PREC_FP32C && sizeof(T) == 8;
    constexpr bool SHIFT = PREC == PREC_FP32C, EXS = BAND && KF == 1;
    constexpr bool FOLD = !BAND;  // the parts are summed apart and added up by k_fold
    __shared__ CT rows_all[4][SEQ_ROWS][33];  // [component or column][leaf]
    __shared__ double sums_all[4][8 + 4 * MAX_KC];
    const TreeView<T>& tv = A.tv;
    const SplitBufs& sp = A.sp;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    auto& rows = rows_all[wib];
    auto& sums = sums_all[wib];
    const int kc = (WHAT == WHAT_DENSITY) ? 0 : A.rec.kc;
    const bool dg = WHAT == WHAT_INTERP && A.rec.need_dg != 0;
    const bool unit = WHAT == WHAT_DENSITY && A.unit_mass != 0;
    // the sums of this lane: component ra of a pair times column rb (-1: none), to field fo of the outputs
    const int nsum = (WHAT == WHAT_DENSITY) ? 1 : 4 + 4 * kc + (dg ? 4 : 0);
    int ra[2], rb[2], fo[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int q = lane + 32 * u;
        ra[u] = 0; rb[u] = -1; fo[u] = -1;
        if (q >= nsum) continue;
        if (q < 4) { ra[u] = q; fo[u] = q; }
        else if (q < 4 + 4 * kc) {
            const int c = (q - 4) >> 2, d = (q - 4) & 3;
            ra[u] = d; rb[u] = SEQ_COMP + c;
            fo[u] = d == 0 ? 8 + c : 8 + sp.kcl + 3 * c + d - 1;
        } else {  // m W, then (m W') d
            const int d = q - 4 - 4 * kc;
            ra[u] = 4 + d; rb[u] = SEQ_COMP + MAX_KC + (d ? 1 : 0);
            fo[u] = 4 + d;
        }
        if (WHAT == WHAT_DENSITY) rb[u] = 1;
    }
    const bool two = nsum > 32;
    unsigned long long n_bodyit = 0;
    // the tiles' lists (seq_all), then the chunks, or (FP32C of double particles) the samples of several parts
    const unsigned n1 = sp.seq_all ? (unsigned)sp.ntiles * 32u : 0u;
    const unsigned nm = min(FOLD ? *sp.top : *sp.mcount, sp.ncap);
    const bool chained = !FOLD && !sp.seq_all && nm >= CHAIN_SAMPLES;  // those of few parts are k_bodies'
    const unsigned nw = gridDim.x * (blockDim.x >> 5);
    for (unsigned i = blockIdx.x * (blockDim.x >> 5) + wib; i < n1 + nm; i += nw) {
        const int32_t c0 = i < n1 ? -1 : (FOLD ? (int32_t)(i - n1) : (int32_t)sp.mlist[i - n1]);
        const uint32_t w0 = i < n1 ? i : sp.own[c0], own = w0 & OWN_IDX;
        if (FOLD && w0 == OWN_NONE) continue;
        const int cn = sp.cnt[own];
        const bool heavy = i >= n1 && (w0 & OWN_HEAVY) != 0;
        if (cn == CNT_DEAD || (cn == CNT_HEAVY) != heavy) continue;  // warp-uniform
        if (chained && !long_chain(sp, c0, w0)) continue;
        const int32_t more = i < n1 && cn == RCAP ? sp.head[own] : -1;  // a list of several parts
        if (!FOLD && more >= 0) continue;
        const int64_t k = sample_of(A.src, sp.tile0 + (own >> 5), own & 31);
        if (k < 0) continue;
        T p[3], dd[3];
        sample_coords(A.src, k, p, dd);
        const T ha = ((const T*)sp.ha)[own];
        const CT sig = (KF == 0) ? inv_pi<CT>() : (CT)tv.sig;
        CT ia = CT(0), sa3 = CT(0), sa4 = CT(0);
        if (ST != ST_SCATTER) {
            ia = CT(1) / (CT)ha;
            sa3 = sig * ia * ia * ia;
            sa4 = sa3 * ia;
        }
        const double kha = tv.Kd * (double)ha;
        const double fa2 = kha * kha;
        const double ika = (KF == 1 && ST != ST_SCATTER) ? 0.5 / (double)ha : 0.0;
        const float qe = (KF == 0) ? 1.f : tv.qedge;
        const size_t q0 = (size_t)(own >> 5) * RCAP * 32 + (own & 31);
        const int64_t first = (SHIFT && cn > 0) ? (int64_t)__float_as_int(sp.ent4[q0].w) + __ffs(sp.emask[q0]) - 1 : 0;
        Acc S[2];
        S[0].zero();
        S[1].zero();
        // the tile's list (not a heavy sample's), then the chunks; with k_fold, one part
        int32_t chunk = (FOLD || heavy) ? c0 : -1;
        while (true) {
            const int n = chunk < 0 ? cn : sp.ccnt[chunk];
            const size_t e0 = chunk < 0 ? q0 : (size_t)sp.ebase + (size_t)chunk * RCAP;
            const int est = chunk < 0 ? 32 : 1;
            const float* esh = !EXS || kc == 0 ? nullptr
                               : chunk < 0 ? sp.eshift + (size_t)(own >> 5) * RCAP * kc * 32 + (own & 31)
                                           : sp.eshift + e0 * kc;
            // lane l: entry l of the part, and the pairs up to it
            float4 en = make_float4(0.f, 0.f, 0.f, 0.f);
            unsigned em = 0;
            if (lane < n) {
                en = sp.ent4[e0 + (size_t)lane * est];
                em = sp.emask[e0 + (size_t)lane * est];
            }
            int upto = __popc(em);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(PSB_FULL, upto, o);
                if (lane >= o) upto += t;
            }
            const int np = __shfl_sync(PSB_FULL, upto, 31);
            for (int w = 0; w < np; w += 32) {
                // lane j: pair w + j of the part, leaf li of entry e
                const int at = w + lane;
                int e = 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    if (__shfl_sync(PSB_FULL, upto, e + o - 1) <= at) e += o;
                unsigned m = __shfl_sync(PSB_FULL, em, e);
                int r = at - (__shfl_sync(PSB_FULL, upto, e) - __popc(m)), bit = 0;  // m's r-th bit
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const int c = __popc(m & ((1u << o) - 1u));
                    if (r >= c) { r -= c; bit += o; m >>= o; }
                }
                const float qx = __shfl_sync(PSB_FULL, en.x, e), qy = __shfl_sync(PSB_FULL, en.y, e),
                            qz = __shfl_sync(PSB_FULL, en.z, e);
                const int64_t li = (int64_t)__shfl_sync(PSB_FULL, __float_as_int(en.w), e) + bit;
                __syncwarp();
                if (at < np) {
                    CT dx, dy, dz, W, c, mr, mb;
                    if constexpr (PREC == PREC_FP64) {
                        const double2 a = __ldg(&tv.leafD[0][li]), b = __ldg(&tv.leafD[1][li]), s = __ldg(&tv.leafD[2][li]);
                        dx = __dsub_rn((double)p[0], a.x);
                        dy = __dsub_rn((double)p[1], a.y);
                        dz = __dsub_rn((double)p[2], b.x);
                        f64_pair_weights<ST, KF>(tv.kern, dx, dy, dz, ia, sa3, b.y, s.x, W, c);
                        mr = s.y;
                        mb = (dg || !unit) ? (CT)__ldg(&tv.m[li]) : CT(1);
                    } else {
                        const float4 L = __ldg(&tv.leaf4[li]), K = __ldg(&tv.leafK[li]);
                        if constexpr (BAND) {
                            dx = __fsub_rn(qx, L.x);
                            dy = __fsub_rn(qy, L.y);
                            dz = __fsub_rn(qz, L.z);
                            f32c_pair_weights<ST, KF>(
                                tv.kern, tv.Kf, qe, dx, dy, dz, ia, sa3, sa4, fa2, ika, (float)ha, K, L.w,
                                [&]() {
                                    const double ex = __dsub_rn(p[0], __ldg(&tv.x[li]));
                                    const double ey = __dsub_rn(p[1], __ldg(&tv.y[li]));
                                    const double ez = __dsub_rn(p[2], __ldg(&tv.z[li]));
                                    return __fma_rn(ex, ex, __fma_rn(ey, ey, __dmul_rn(ez, ez)));
                                },
                                [&]() { return __dmul_rn(tv.Kd, __ldg(&tv.h[li])); }, W, c);
                        } else {
                            dx = __fsub_rn(p[0], L.x);
                            dy = __fsub_rn(p[1], L.y);
                            dz = __fsub_rn(p[2], L.z);
                            f32_pair_weights<ST, KF>(tv.kern, ex_d2_pp<T>(p, L.x, L.y, L.z), ia, sa3, sa4, K.x, K.y, W, c);
                        }
                        mr = K.w;
                        mb = (dg || !unit) ? __ldg(&tv.mf[li]) : 1.f;
                    }
                    if (WHAT == WHAT_DENSITY) {
                        rows[0][lane] = W;
                        rows[1][lane] = unit ? CT(1) : mb;
                    } else {
                        const CT gc = acc_mul(mr, c);
                        rows[0][lane] = acc_mul(mr, W);
                        rows[1][lane] = acc_mul(gc, dx);
                        rows[2][lane] = acc_mul(gc, dy);
                        rows[3][lane] = acc_mul(gc, dz);
                        if (dg) {
                            const CT mc = acc_mul(mb, c);
                            rows[4][lane] = W;
                            rows[5][lane] = dx;
                            rows[6][lane] = dy;
                            rows[7][lane] = dz;
                            rows[SEQ_COMP + MAX_KC][lane] = mb;
                            rows[SEQ_COMP + MAX_KC + 1][lane] = mc;
                        }
                        for (int s = 0; s < kc; ++s) {
                            CT a;
                            if constexpr (EXS) a = __fadd_rn(__ldg(&A.colR[s][li]), esh[(e * kc + s) * est]);
                            else if constexpr (SHIFT) a = __fsub_rn(__ldg(&A.colF[s][li]), __ldg(&A.colF[s][first]));
                            else a = (CT)__ldg(&A.colT[s][li]);
                            rows[SEQ_COMP + s][lane] = a;
                        }
                    }
                }
                __syncwarp();
                ++n_bodyit;
                const int nj = min(32, np - w);
#pragma unroll 4
                for (int j = 0; j < nj; ++j) {
                    const CT v = rows[ra[0]][j];
                    if (rb[0] < 0) S[0].add(v);
                    else acc_mac(S[0], rows[rb[0]][j], v);
                    if (two) {
                        const CT v1 = rows[ra[1]][j];
                        if (rb[1] < 0) S[1].add(v1);
                        else acc_mac(S[1], rows[rb[1]][j], v1);
                    }
                }
            }
            if (FOLD || i < n1) break;
            chunk = chunk < 0 ? c0 : sp.next[chunk];
            if (chunk < 0) break;
        }
        if (FOLD && (chunk >= 0 || more >= 0)) {  // a part, for k_fold
            double* o = sp.part + (chunk >= 0 ? chunk : (size_t)sp.ncap + more);
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (fo[u] >= 0) o[fo[u] * 2 * (size_t)sp.ncap] = S[u].get();
            continue;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (fo[u] >= 0) sums[fo[u]] = S[u].get();
        __syncwarp();
        if (lane == 0) {
            if (WHAT == WHAT_DENSITY) {
                A.out[0][k] = (PREC == PREC_FP64) ? (T)sums[0] : (T)(CT)sums[0];
            } else {
                PlainD S1, G[3], Dm, Dg[3], Sw[MAX_KC], Sg[MAX_KC][3];
                double a0[MAX_KC];
                S1.s = sums[0];
                Dm.s = dg ? sums[4] : 0.0;
                for (int d = 0; d < 3; ++d) {
                    G[d].s = sums[1 + d];
                    Dg[d].s = dg ? sums[5 + d] : 0.0;
                }
                for (int c = 0; c < MAX_KC; ++c) {
                    const bool on = c < kc;
                    Sw[c].s = on ? sums[8 + c] : 0.0;
                    for (int d = 0; d < 3; ++d) Sg[c][d].s = on ? sums[8 + sp.kcl + 3 * c + d] : 0.0;
                    a0[c] = (!on || !SHIFT || cn == 0) ? 0.0 : (EXS ? (double)A.colT[c][first] : (double)A.colF[c][first]);
                }
                write_interp_outputs<T, PlainD, CT, MAX_KC>(A, k, S1, G, Sw, Sg, Dm, Dg, a0);
            }
        }
        __syncwarp();
    }
    if (lane == 0 && A.stats && n_bodyit) atomicAdd(&A.stats[5], n_bodyit);
}

}  // namespace psb
