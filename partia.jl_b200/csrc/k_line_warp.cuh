// k_line_warp.cuh -- line integrals of double particles: one warp per line, and
// tiles of 32 lines that run together.
//
// k_line_warp: lines that do not run together (sight lines in any direction, but
// see k_line_share), and calls of too few tiles to fill the GPU, where the tile
// kernel's union walk visits far more than any one line needs, or leaves most
// SMs idle.  The warp walks the
// tree for its line 32 nodes at a time (window_walk) and takes a span's leaves
// one per lane, with the exact inclusion test; each sum then runs through the
// accepted leaves in leaf order in a lane of its own, so a line's bits are
// those of the tile kernel.  Double particles only: with float ones the line
// distance cancels to noise of the size of h^2, and the neighbours depend on
// the reference's pruning of every single node.
#pragma once

#include "k_split.cuh"

namespace psb {

// Bound by issue: about 60 instructions per 32 nodes, 100 per span and 8 per
// pair.  20,011 sight lines through 300k clump particles (M5, FP64, two
// scalars): 79 ms in tiles of 32, a call takes 3.5 ms with this.
template <int PREC, int ST>
__global__ void __launch_bounds__(128, 8) k_line_warp(const __grid_constant__ Args<double> A) {
    using T = double;
    using CT = typename std::conditional<PREC == PREC_FP64, double, float>::type;
    using Acc = typename std::conditional<PREC == PREC_FP64, PlainD, KahanF>::type;
    constexpr bool F32C = PREC == PREC_FP32C;  // float distances relative to the span
    __shared__ int32_t q_all[4][WQ];
    __shared__ CT rows_all[4][1 + MAX_KC][33];  // [w, columns][leaf]
    __shared__ double sums_all[4][1 + MAX_KC];
    const TreeView<T>& tv = A.tv;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    auto& rows = rows_all[wib];
    const int64_t item = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    int64_t line = item;  // tile * 32 + lane
    if (A.tile_list) {  // groups of lines that k_line_tile handed over (tile_lines each)
        const int64_t at = item / A.tile_lines;
        if (at >= (int64_t)*A.tile_count) return;
        line = (int64_t)A.tile_list[at] * A.tile_lines + item % A.tile_lines;
    }
    if ((line >> 5) >= A.src.ntiles) return;
    const int64_t k = sample_of(A.src, line >> 5, (int)(line & 31));
    if (k < 0) return;  // warp-uniform
    T o[3], m[3];
    sample_coords(A.src, k, o, m);
    const float of[3] = {(float)o[0], (float)o[1], (float)o[2]};
    const float mf3[3] = {(float)m[0], (float)m[1], (float)m[2]};
    const double od[3] = {(double)o[0], (double)o[1], (double)o[2]}, md[3] = {(double)m[0], (double)m[1], (double)m[2]};
    const float onorm = fabsf(of[0]) + fabsf(of[1]) + fabsf(of[2]);
    const float S = tv.coord_err / U1;
    const float el = 4.f * U1 * (onorm + 6.f * S) + 1e-18f;
    // the float node test needs a unit direction and floats that do not
    // overflow; other lines take the reference's arithmetic
    const double mm = md[0] * md[0] + md[1] * md[1] + md[2] * md[2];
    const bool plain = line_plain(od, mm);
    T ha = T(0);
    if (ST != ST_SCATTER) ha = (A.hmode == PSB_H_PER_SAMPLE) ? A.hs[k] : A.hs[0];
    const T Kt = (T)tv.Kd;
    const T ra = X<T>::mul(Kt, ha);
    const T ra2 = X<T>::mul(ra, ra);
    const float ra2_hi = (ST == ST_SCATTER) ? 0.f : __double2float_ru((double)ra2) * (1.f + RELM) + 1e-36f;
    // the rounding of the exact distance D^2 - (D.m)^2, which cancels
    const float e64 = 4.5e-16f * (onorm + 6.f * S) * (onorm + 6.f * S) + 1e-36f;
    const CT ia = (ST != ST_SCATTER) ? CT(1) / (CT)ha : CT(0);
    const int kc = A.rec.kc;
    const int nlut = A.lut_n;
    const bool short_lut = nlut == LUT_SHORT_N;
    auto lutv = [&](int i) -> CT {
        if constexpr (PREC == PREC_FP64) return short_lut ? (CT)__ldg(&A.lut_fs[i]) : __ldg(&A.lut_d[i]);
        else return __ldg(short_lut ? &A.lut_fs[i] : &A.lut_f[i]);
    };
    const CT Kc = (CT)tv.Kd;
    const CT idq = CT(1) / (CT)(tv.Kd / (double)(nlut - 1));
    Acc sum;  // lane 0: S1, lane 1 + c: Sw_c
    sum.zero();
    unsigned n_pairs = 0;
    uint32_t steps = 0;

    auto node_ok = [&](int ni) -> bool {
        if (plain) {
            const float4 lo = __ldg(&tv.node_lo[ni]), hi = __ldg(&tv.node_hi[ni]);
            return !(lb_d2_line_box(of, mf3, el, lo, hi) > hi_r2_node<ST>(ra2_hi, lo.w, tv.Kf) + e64);
        }
        const T d2n = ex_d2_line_box<T>(o, m, tv, ni);
        return !(d2n > ((ST == ST_GATHER) ? ra2 : ex_r2<ST, T>(ra2, __ldg(&tv.nscale[ni]), Kt)));
    };
    auto span_fn = [&](int32_t id) {
        int64_t lo;
        int cnt;
        if (id >= (int32_t)tv.n) {
            lo = (int64_t)id - tv.n;
            cnt = 1;
        } else {
            const int4 lk = __ldg(&tv.links[id - 1]);
            lo = (int64_t)lk.z - 1;
            cnt = lk.w - lk.z + 1;
        }
        const int64_t li = lo + lane;
        // in float first: most spans' leaves all miss the line
        float cf[3];
        const float cerr = line_perp(od, md, (double)__ldg(&tv.x[lo]), (double)__ldg(&tv.y[lo]), (double)__ldg(&tv.z[lo]), cf);
        float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
        bool maybe = false;
        if (lane < cnt) {
            L = __ldg(&tv.leaf4[li]);
            const float ev = 8.f * U1 * (2.f * __ldg(&tv.spanb[lo]).x + fabsf(cf[0]) + fabsf(cf[1]) + fabsf(cf[2])) * (1.f + 4.f * U1) +
                             cerr + 1e-18f;
            const float kb = tv.Kf * L.w;
            const float r2 = (ST == ST_GATHER) ? ra2_hi : fmaxf(ra2_hi, kb * kb * (1.f + 2.f * RELM) + 1e-36f);
            const float reach = sqrtf(r2 + e64) * (1.f + RELM) + ev;
            maybe = !plain || line_fs_f32(L, cf, mf3) * (1.f - RELM) <= reach * reach * (1.f + RELM);
        }
        if (!__any_sync(PSB_FULL, maybe)) return;
        bool in = false;
        T e2 = T(0);
        if (maybe) {
            e2 = ex_d2_line<T>(o, m, __ldg(&tv.x[li]), __ldg(&tv.y[li]), __ldg(&tv.z[li]));
            in = e2 <= ex_r2<ST, T>(ra2, __ldg(&tv.h[li]), Kt);
        }
        const unsigned acc = __ballot_sync(PSB_FULL, in);
        if (!acc) return;
        n_pairs += __popc(acc);
        if (in) {
            CT dr, ib, mr;
            if constexpr (F32C) {
                dr = line_r_f32(L, cf, mf3);
                ib = __ldg(&tv.leafK[li]).x;
                mr = __ldg(&tv.mrho[li]);
            } else {
                dr = line_r_f64(e2);
                ib = __ldg(&tv.leafD[1][li]).y;
                mr = __ldg(&tv.leafD[2][li]).y;
            }
            rows[0][lane] = acc_mul(mr, line_pair_W<ST, CT>(dr, ia, ib, lutv, idq, nlut, Kc));
            for (int c = 0; c < kc; ++c) {
                if constexpr (F32C) rows[1 + c][lane] = __ldg(&A.colF[c][li]);
                else rows[1 + c][lane] = __ldg(&A.colT[c][li]);
            }
        }
        __syncwarp();
        if (lane <= kc) {
#pragma unroll 4
            for (unsigned b = acc; b; b &= b - 1) {
                const int j = __ffs(b) - 1;
                const CT w = rows[0][j];
                if (lane == 0) sum.add(w);
                else acc_mac(sum, rows[lane][j], w);
            }
        }
        __syncwarp();
    };
    const bool ok = window_walk<true>(tv, q_all[wib], node_ok, span_fn, steps);

    if (lane <= kc) sums_all[wib][lane] = sum.get();
    __syncwarp();
    if (lane == 0) {
        PlainD S1, Sw[MAX_KC];
        S1.s = sums_all[wib][0];
        for (int c = 0; c < MAX_KC; ++c) Sw[c].s = c < kc ? sums_all[wib][1 + c] : 0.0;
        write_line_outputs<T, PlainD, MAX_KC>(A, k, S1, Sw);
        if (A.stats) {
            atomicAdd(&A.stats[0], (unsigned long long)n_pairs);
            atomicAdd(&A.stats[2], (unsigned long long)steps);
        }
        if (!ok) atomicOr(A.err, PSB_DERR_TRAVERSAL);
    }
}

// A tile of 32 lines takes one walk together if all pass within LINE_TUBE mean
// particle spacings of one of them inside the particles' box; the lines of
// another tile go to k_line_warp.  (Parallel beams always run together.)
constexpr double LINE_TUBE = 1.0;

// Where the lines of a tile meet much the same spans whatever their directions
// (a small set, large supports), all tiles take their lines together: FP64 here
// with G = 1, FP32C in k_lines.  A warp per line pays for every span its line
// meets, a tile for the spans that any of its lines meets, and a tile lasts as
// long as its walk whether others run beside it or not.  So the tiles are taken
// from a share of (spans of a line) / (spans of its tile) on, of 16 tiles and 64
// spans, and of that share times the tiles (calls of so few tiles that no share
// below 0.9 is enough are not asked about).  Lines in any direction, ms a call,
// a warp per line and tiles:
//                                share     FP64, 100,000 / 500,000 lines      FP32C
//   Plummer   1000 particles, M4  0.74      3.1   1.0    14.0   3.2       3.0   0.8    13.6  2.4
//   Plummer   5000, M6            0.57      8.8   3.6    41.6  14.1       8.7   3.0    40.8 10.3
//   Plummer 30,000, M6            0.27     16.9  17.3    80.9  66.6      16.8  14.0    80.6 50.0
//   Plummer 30,000, M4            0.18      9.6  13.7    45.8  51.5       9.6  12.0    45.5 41.5
//   clumps  30,000, M6            0.19      9.9  10.0    46.9  40.8       9.7   6.6    45.6 23.2
//   clumps  30,000, M4            0.15      6.0   8.8    27.8  35.4       5.8   5.4    26.9 18.6
//   uniform 30,000, M6            0.12      7.9  14.0    37.4  55.8       7.8  11.7    36.9 42.2
// and 20,000 lines through the second: 2.2 2.5 (FP64), 2.1 1.9.  (G = 8 takes 1.9
// to 2.5 times the time of G = 1 on lines apart.)
constexpr float LINE_SHARE_FP64 = 0.185f, LINE_SHARE_TILES_FP64 = 600.f;
constexpr float LINE_SHARE_FP32C = 0.14f, LINE_SHARE_TILES_FP32C = 400.f;
constexpr int SHARE_THREADS = 512;
template <int ST>
__global__ void __launch_bounds__(SHARE_THREADS)
    k_line_share(const __grid_constant__ Args<double> A, const int32_t* parent, float least, float tiles,
                 unsigned* together) {
    const TreeView<double>& tv = A.tv;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ float4 lo_s[64], hi_s[64];
    __shared__ int line_s[SHARE_THREADS / 32], tile_s[SHARE_THREADS / 32];
    if (threadIdx.x < 64) {  // the box of a leaf's span, and its largest h
        const int64_t b = (tv.n - 1) * threadIdx.x / 63;
        const float x = (float)tv.x[b], y = (float)tv.y[b], z = (float)tv.z[b];
        float4 lo = make_float4(x, y, z, (float)tv.h[b]), hi = lo;
        for (int32_t p = parent[tv.n + b - 1]; p > 0; p = parent[p - 1]) {
            const int4 lk = tv.links[p - 1];
            if (lk.w - lk.z >= SPAN) break;
            lo = tv.node_lo[p - 1];
            hi = tv.node_hi[p - 1];
        }
        lo_s[threadIdx.x] = lo;
        hi_s[threadIdx.x] = hi;
    }
    __syncthreads();
    // a warp takes a tile, a line per lane
    const int64_t k = sample_of(A.src, (A.src.ntiles - 1) * warp / (SHARE_THREADS / 32 - 1), lane);
    double o[3] = {0.0, 0.0, 0.0}, m[3] = {0.0, 0.0, 1.0}, ha = 0.0;
    if (k >= 0) {
        sample_coords(A.src, k, o, m);
        if (ST != ST_SCATTER) ha = (A.hmode == PSB_H_PER_SAMPLE) ? A.hs[k] : A.hs[0];
    }
    const float of[3] = {(float)o[0], (float)o[1], (float)o[2]}, mf[3] = {(float)m[0], (float)m[1], (float)m[2]};
    const float ra = tv.Kf * (float)ha;
    int by_line = 0, by_tile = 0;
    for (int i = 0; i < 64; ++i) {
        const float4 lo = lo_s[i];
        const unsigned met = __ballot_sync(
            PSB_FULL, k >= 0 && lb_d2_line_box(of, mf, 0.f, lo, hi_s[i]) <= hi_r2_node<ST>(ra * ra, lo.w, tv.Kf));
        by_line += __popc(met);
        by_tile += met != 0;
    }
    if (lane == 0) { line_s[warp] = by_line; tile_s[warp] = by_tile; }
    __syncthreads();
    if (threadIdx.x == 0) {
        int l = 0, t = 0;
        for (int w = 0; w < SHARE_THREADS / 32; ++w) { l += line_s[w]; t += tile_s[w]; }
        const float share = (float)l / (32.f * (float)max(t, 1));
        *together = share >= least && share * (float)A.src.ntiles >= tiles;
    }
}

// Per-warp shared memory: the leaves of a span that reach the tile.
template <class CT, int KC> struct TStage {
    float4 L[SPAN];   // offset from the span's first leaf, h
    float2 AB[SPAN];  // squared radius thresholds: surely in below A, surely out above B
    CT ih[SPAN];      // 1/h
    CT mr[SPAN];      // m/rho
    CT col[KC][SPAN];
    uint8_t j[SPAN];  // index in the span
    int32_t q[WQ];
};

// Line integrals of double particles over tiles of 32 lines that run
// together, one line per lane.  The walk and a first test of a span's leaves
// (one per lane) take the tile's lines as a tube around one of them; the
// leaves that reach the tube are packed in shared memory, each lane builds
// the mask of those within reach of its own line (float distances against one
// error band per span, the exact test for undecided pairs), and then sums its
// own pairs, in leaf order.  Bound by issue.  Testing every leaf of a span
// against every line, with a square root before the decision and a divergent
// sum behind it, took 4.5e9 warp instructions for 2M clump particles on a
// 512^2 beam; this takes 2.4e9 (k_beam_tile_cost for the times).
//
// G = 1: a warp takes a tile, one line per lane.  G = 8: a warp takes four of
// a tile's lines, eight lanes each (every eighth leaf, every eighth pair, the
// sums in order in every lane): about 1.5 times the instructions, at an eighth
// of the time for the longest line.  It serves calls of few tiles.
template <int PREC, int ST, int KC, int G>
__global__ void __launch_bounds__(128, KC <= 1 ? 8 : 6) k_line_tile(const __grid_constant__ Args<double> A) {
    using CT = typename std::conditional<PREC == PREC_FP64, double, float>::type;
    using Acc = typename std::conditional<PREC == PREC_FP64, PlainD, KahanF>::type;
    constexpr bool F32C = PREC == PREC_FP32C;
    __shared__ TStage<CT, KC> stage_all[4];
    const TreeView<double>& tv = A.tv;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    auto& st = stage_all[wib];
    const int64_t wid = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    int64_t tile = wid / G;
    if (tile >= (A.tile_count ? min((int64_t)*A.tile_count, A.src.ntiles) : A.src.ntiles)) return;
    // explicit lines, all tiles together: k_lines' (FP32C), or those of G = 1 where both are launched
    if (A.sp.ovf_count && (A.sp.ovf_count[1] ? F32C || G > 1 : A.tile_lines == 4 && G == 1)) return;
    if (A.tile_list) tile = A.tile_list[tile];  // heavy first, or the heavy ones
    if (A.tile_cost && A.tile_cost[2 * tile] < 0.f) return;  // handed over
    // lane g of the G lanes of this warp's line lane / G
    const int g = lane % G;
    const int64_t k = sample_of(A.src, tile, G == 1 ? lane : (int)(wid % G) * (32 / G) + lane / G);
    const bool valid = k >= 0;
    if (G > 1 && !__any_sync(PSB_FULL, valid)) return;
    double o[3] = {0.0, 0.0, 0.0}, m[3] = {0.0, 0.0, 1.0};
    if (valid) sample_coords(A.src, k, o, m);
    // the tube: all lines within Rt of line c inside the particles' box
    const unsigned vm = __ballot_sync(PSB_FULL, valid);
    const int c = (G == 1 && ((vm >> 12) & 1u)) ? 12 : __ffs(vm) - 1;  // pixel (4, 1) of a full 8 x 4 tile
    double oc[3], mc[3];
    float Rt;
    {
        double t = 0.0, mm = 0.0, e = 0.0, e2 = 0.0, a[3];
        for (int d = 0; d < 3; ++d) {
            t += (A.line_centre[d] - o[d]) * m[d];
            mm += m[d] * m[d];
        }
        for (int d = 0; d < 3; ++d) a[d] = o[d] + t * m[d];
        for (int d = 0; d < 3; ++d) {
            oc[d] = __shfl_sync(PSB_FULL, o[d], c);
            mc[d] = __shfl_sync(PSB_FULL, m[d], c);
            const double da = a[d] - __shfl_sync(PSB_FULL, a[d], c), dm = m[d] - mc[d];
            e += da * da;
            e2 += dm * dm;
        }
        const double r = (sqrt(e) + A.line_extent * sqrt(e2)) * (1.0 + 1e-12);
        if (A.sp.ovf_count) {
            // (a line's limits are those of the float tests, k_line_warp's `plain`)
            const bool near = (r <= A.line_tube || A.sp.ovf_count[1]) && line_plain(o, mm);
            if (!__all_sync(PSB_FULL, !valid || near)) {
                if (lane == 0) list_lines(A, G == 1 ? tile : wid, G);
                return;
            }
        }
        Rt = __uint_as_float(__reduce_max_sync(PSB_FULL, valid ? __float_as_uint(__double2float_ru(r)) : 0u)) * (1.f + 2.f * U1);
    }
    const float ocf[3] = {(float)oc[0], (float)oc[1], (float)oc[2]};
    const float mcf[3] = {(float)mc[0], (float)mc[1], (float)mc[2]};
    const float mf3[3] = {(float)m[0], (float)m[1], (float)m[2]};
    // |o|_1 (the tile's largest) and the particle coordinate scale S (coord_err = 2^-23 S)
    const float onorm = __uint_as_float(__reduce_max_sync(
        PSB_FULL, valid ? __float_as_uint((float)(fabs(o[0]) + fabs(o[1]) + fabs(o[2])) * (1.f + 2.f * U1)) : 0u));
    const float S = tv.coord_err / U1;
    const float el = 4.f * U1 * (onorm + 6.f * S) + 1e-18f;
    const float e64 = 4.5e-16f * (onorm + 6.f * S) * (onorm + 6.f * S) + 1e-36f;
    double ha = 0.0;
    if (ST != ST_SCATTER && valid) ha = (A.hmode == PSB_H_PER_SAMPLE) ? A.hs[k] : A.hs[0];
    const double ra = X<double>::mul(tv.Kd, ha);
    const double ra2 = X<double>::mul(ra, ra);
    const bool takes = valid && (ST == ST_SCATTER || ra2 == ra2);  // (a radius of NaN: no neighbours)
    float ra2_hi = 0.f, ra2_lo = 0.f, ra2max = 0.f;
    if (ST != ST_SCATTER) {
        ra2_hi = __double2float_ru(ra2) * (1.f + RELM) + 1e-36f;
        ra2_lo = __double2float_rd(ra2) * (1.f - RELM);
        ra2max = __uint_as_float(__reduce_max_sync(PSB_FULL, valid && ra2_hi > 0.f ? __float_as_uint(ra2_hi) : 0u));
    }
    const CT ia = (ST != ST_SCATTER) ? CT(1) / (CT)ha : CT(0);
    const int kc = A.rec.kc;
    const int nlut = A.lut_n;
    const bool short_lut = nlut == LUT_SHORT_N;
    // The table is read from global memory: one copy in each SM's L1 serves every CTA there.
    auto lutv = [&](int i) -> CT {
        if constexpr (PREC == PREC_FP64) return short_lut ? (CT)__ldg(&A.lut_fs[i]) : __ldg(&A.lut_d[i]);
        else return __ldg((short_lut ? A.lut_fs : A.lut_f) + i);
    };
    const CT Kc = (CT)tv.Kd;
    const CT idq = CT(1) / (CT)(tv.Kd / (double)(nlut - 1));
    Acc S1, Sw[KC];
    S1.zero();
#pragma unroll
    for (int q = 0; q < KC; ++q) Sw[q].zero();
    unsigned n_pairs = 0, n_retest = 0;
    uint32_t steps = 0;

    auto node_ok = [&](int ni) -> bool {
        const float4 lo = __ldg(&tv.node_lo[ni]), hi = __ldg(&tv.node_hi[ni]);
        return !(lb_d2_line_box(ocf, mcf, el, lo, hi, Rt) > hi_r2_node<ST>(ra2max, lo.w, tv.Kf) + e64);
    };
    auto span_fn = [&](int32_t id) {
        int64_t lo;
        int cnt;
        if (id >= (int32_t)tv.n) {
            lo = (int64_t)id - tv.n;
            cnt = 1;
        } else {
            const int4 lk = __ldg(&tv.links[id - 1]);
            lo = (int64_t)lk.z - 1;
            cnt = lk.w - lk.z + 1;
        }
        const double ax = __ldg(&tv.x[lo]), ay = __ldg(&tv.y[lo]), az = __ldg(&tv.z[lo]);
        const float sbx = __ldg(&tv.spanb[lo]).x;
        // lane j: leaf j against the tube
        float cc[3];
        const float ccerr = line_perp(oc, mc, ax, ay, az, cc);
        const float ec = 8.f * U1 * (2.f * sbx + fabsf(cc[0]) + fabsf(cc[1]) + fabsf(cc[2])) * (1.f + 4.f * U1) + ccerr + 1e-18f;
        float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
        float rlo2 = 0.f, rhi2 = 0.f;  // squared radius bounds of the leaf
        bool keep = false;
        if (lane < cnt) {
            L = __ldg(&tv.leaf4[lo + lane]);
            const float kb = tv.Kf * L.w, rb2 = kb * kb;
            if (ST != ST_GATHER) {
                rlo2 = rb2 * (1.f - 2.f * RELM);
                rhi2 = rb2 * (1.f + 2.f * RELM) + 1e-36f;
            }
            const float reach = sqrtf((ST == ST_SCATTER ? rhi2 : fmaxf(ra2max, rhi2)) + e64) * (1.f + RELM) + Rt + ec;
            keep = line_fs_f32(L, cc, mcf) * (1.f - RELM) <= reach * reach * (1.f + RELM);
        }
        const unsigned kept = __ballot_sync(PSB_FULL, keep);
        if (!kept) return;
        const int ns = __popc(kept);
        // this lane's line: perpendicular offset of the span's first leaf, and
        // one error band for the span's leaves and the tile's lines
        float cf[3];
        const float cerr = line_perp(o, m, ax, ay, az, cf);
        float E = 8.f * U1 * (2.f * sbx + fabsf(cf[0]) + fabsf(cf[1]) + fabsf(cf[2])) * (1.f + 4.f * U1) + cerr + 1e-18f;
        E = __uint_as_float(__reduce_max_sync(PSB_FULL, valid ? __float_as_uint(E) : 0u));
        auto inner = [&](float r2) {  // (sqrt(r2 - e64) - E)^2, rounded down
            const float r = fmaxf(sqrtf(fmaxf(r2 - e64, 0.f)) * (1.f - RELM) - E, 0.f);
            return r * r * (1.f - RELM);
        };
        auto outer = [&](float r2) {  // (sqrt(r2 + e64) + E)^2, rounded up
            const float r = sqrtf(r2 + e64) * (1.f + RELM) + E;
            return r * r * (1.f + RELM);
        };
        __syncwarp();
        if (keep) {
            const int64_t li = lo + lane;
            const int at = __popc(kept & below);
            st.L[at] = L;
            st.j[at] = (uint8_t)lane;
            if (ST != ST_GATHER) st.AB[at] = make_float2(inner(rlo2), outer(rhi2));
            if constexpr (PREC == PREC_FP64) {
                st.ih[at] = __ldg(&tv.leafD[1][li]).y;
                st.mr[at] = __ldg(&tv.leafD[2][li]).y;
            } else {
                st.ih[at] = __ldg(&tv.leafK[li]).x;
                st.mr[at] = __ldg(&tv.mrho[li]);
            }
#pragma unroll
            for (int q = 0; q < KC; ++q)
                if (q < kc) {
                    if constexpr (PREC == PREC_FP64) st.col[q][at] = __ldg(&A.colT[q][li]);
                    else st.col[q][at] = __ldg(&A.colF[q][li]);
                }
        }
        float As = 0.f, Bs = 0.f;
        if (ST != ST_SCATTER) {
            As = inner(ra2_lo);
            Bs = outer(ra2_hi);
        }
        __syncwarp();
        unsigned acc = 0, maybe = 0;
        if (takes) {
#pragma unroll 4
            for (int j = g; j < ns; j += G) {
                const float fs = line_fs_f32(st.L[j], cf, mf3);
                float At = As, Bt = Bs;
                if (ST != ST_GATHER) {
                    const float2 ab = st.AB[j];
                    At = (ST == ST_SCATTER) ? ab.x : fmaxf(As, ab.x);
                    Bt = (ST == ST_SCATTER) ? ab.y : fmaxf(Bs, ab.y);
                }
                acc |= (unsigned)(fs < At) << j;
                maybe |= (unsigned)(fs <= Bt) << j;
            }
            for (unsigned u = maybe & ~acc; u; u &= u - 1) {  // undecided: the reference's double test
                const int j = __ffs(u) - 1;
                const int64_t li = lo + st.j[j];
                ++n_retest;
                const double e2 = ex_d2_line<double>(o, m, __ldg(&tv.x[li]), __ldg(&tv.y[li]), __ldg(&tv.z[li]));
                if (e2 <= ex_r2<ST, double>(ra2, __ldg(&tv.h[li]), tv.Kd)) acc |= 1u << j;
            }
            n_pairs += __popc(acc);
        }
        auto weight = [&](int j) -> CT {
            CT dr;
            if constexpr (PREC == PREC_FP64) {
                const int64_t li = lo + st.j[j];
                dr = line_r_f64(ex_d2_line<double>(o, m, __ldg(&tv.x[li]), __ldg(&tv.y[li]), __ldg(&tv.z[li])));
            } else {
                dr = line_r_f32(st.L[j], cf, mf3);
            }
            return acc_mul(st.mr[j], line_pair_W<ST, CT>(dr, ia, st.ih[j], lutv, idq, nlut, Kc));
        };
        if constexpr (G == 1) {
            for (; acc; acc &= acc - 1) {
                const int j = __ffs(acc) - 1;
                const CT w = weight(j);
                S1.add(w);
#pragma unroll
                for (int q = 0; q < KC; ++q)
                    if (q < kc) acc_mac(Sw[q], st.col[q][j], w);
            }
        } else {
#pragma unroll
            for (int q = 1; q < G; q <<= 1) acc |= __shfl_xor_sync(PSB_FULL, acc, q);
            while (__any_sync(PSB_FULL, acc != 0)) {
                // lane g takes the line's g-th pair of those left
                unsigned b = acc;
                for (int q = 0; q < g; ++q) b &= b - 1;
                const int j = b ? __ffs(b) - 1 : 0;
                CT w = CT(0);
                if (b) w = weight(j);
                const int np = min(G, __popc(acc));
#pragma unroll
                for (int q = 0; q < G; ++q) {
                    const int from = (lane & ~(G - 1)) + q;
                    const CT wq = __shfl_sync(PSB_FULL, w, from);
                    const int jq = __shfl_sync(PSB_FULL, j, from);
                    if (q < np) {
                        S1.add(wq);
#pragma unroll
                        for (int t = 0; t < KC; ++t)
                            if (t < kc) acc_mac(Sw[t], st.col[t][jq], wq);
                    }
                }
#pragma unroll
                for (int q = 0; q < G; ++q) acc &= acc - 1;
            }
        }
    };
    const bool ok = window_walk<true>(tv, st.q, node_ok, span_fn, steps);

    if (valid && g == 0) write_line_outputs<double, Acc, KC>(A, k, S1, Sw);
    unsigned long long t_pairs = n_pairs, t_retest = n_retest;
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) {
        t_pairs += __shfl_xor_sync(PSB_FULL, t_pairs, q);
        t_retest += __shfl_xor_sync(PSB_FULL, t_retest, q);
    }
    if (lane == 0 && A.stats) {
        atomicAdd(&A.stats[0], t_pairs);
        atomicAdd(&A.stats[1], t_retest);
        atomicAdd(&A.stats[2], (unsigned long long)steps);
    }
    if (!ok && lane == 0) atomicOr(A.err, PSB_DERR_TRAVERSAL);
}

}  // namespace psb
