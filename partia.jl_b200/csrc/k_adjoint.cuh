// k_adjoint.cuh -- adjoint (vector-Jacobian product) kernels for every kernel
// family: M4's f'/q and its q-derivative are written out below (m4_wce), the
// others' come from kern_g12; the Hessian is used in products with vectors only
// and never formed.  The support K enters every radius rule.
//
// For a loss L = sum_s sum_k gout_k(s) out_k(s) the forward pass in FP64 first
// writes, per sample, the cotangents lambda of its sums (S1, G, Dm, Dg, Sw_c,
// Sg_c; write_sum_cotangents).  The kernels here then sum the pair terms per
// PARTICLE, so that every gradient is accumulated by one thread and no float
// atomics are needed:
//   dL/dm_b   = sum_s (aS W + aG.gradW) / rho_b + lDm W + lDg.gradW
//   dL/dA_c,b = sum_s m_b/rho_b (lSw_c W + lSg_c.gradW)
//   dL/dx_b   = -sum_s m_b/rho_b (aS gradW + H aG) + m_b (lDm gradW + H lDg)
// with aS = lS1 + sum_c lSw_c A_c,b, aG = lG + sum_c A_c,b lSg_c, W, gradW and
// the Hessian H of the kernel at delta = x_s - x_b (averaged over h_a and h_b
// in the symmetric strategy).  Densities and smoothing lengths are held fixed
// (h_a from the nearest particle is piecewise constant in the positions).
//
// Point samples: one warp per 32 Morton-consecutive particles walks a second
// LBVH built over the samples (node scale = subtree max of h_a) with the
// forward's radius rules seen from the particle, and re-decides every pair
// with the forward's exact arithmetic, so the pair set is the forward's.
// Parallel-beam lines: the pixels whose lines can pass within a particle's
// support (the particle projected onto the frame plane) are visited by a
// lane, eight lanes or a warp, after their number, and each pair is re-decided
// with the forward's line distance.
#pragma once

#include "k_points.cuh"

namespace psb {

// Pair lists of the two-kernel adjoint: one chain of blocks per tile of 32
// particles, taken from a pool with an atomic counter.  A block holds up to
// ADJ_CH entries per lane; an entry is a span of the sample tree (its first
// sample) and the mask of the samples that pair with the lane's particle.
// The warp takes a new block when any lane's is full, so where a chain's
// blocks begin and end follows from the walk alone.  A tile for which the
// pool runs out is marked and listed (the host grows the pool and walks
// again).
constexpr int ADJ_CH = 16;
struct AdjLists {
    uint2* ent;           // [block][ADJ_CH][32]: (first sample of the span, mask)
    uint8_t* bcnt;        // [block][32]: entries of each lane in the block
    int32_t* bnext;       // [block]: the tile's next block, -1 after its last
    int32_t* btile;       // [block]: the block's tile
    double* part;         // [block][AdjAcc::NF][32]: the block's partial sums
    int32_t* head;        // [tile]: first block, -1 without pairs, -2 overflowed
    unsigned* top;        // blocks taken
    int64_t nblocks;      // pool size
    int32_t* ovf_tiles;   // overflowed tiles
    unsigned* ovf_count;
};

struct AdjArgs {
    TreeView<double> pt;          // particles (Morton order)
    TreeView<double> sv;          // samples, in the order of their own LBVH; h = h_a
    const double* colT[MAX_KC];   // the catalog's distinct columns (particle Morton order)
    int kc;
    const double* lam;            // sum cotangents [q][sample] (sample-tree order for points)
    int64_t lam_stride;
    const int64_t* porder;        // particle Morton position -> caller's index
    double* gm;
    double* gx;
    double* gy;
    double* gz;
    double* gcol[MAX_KC];         // gradient of catalog column c (caller's order), may be null
    // parallel-beam lines
    SampleSrc<double> beam;
    int hmode;
    const double* hs;
    double ha_max;
    const double* lut;
    unsigned* err;
    unsigned long long* stats;    // [0] pairs, [2] walk steps
    // the two-kernel point path (k_adj_points' list form, k_adj_bodies, k_adj_combine)
    AdjLists al;
    const double* lamT;           // records of the samples for k_adj_bodies (AdjRec, sample-tree order)
    const int32_t* tile_list;     // k_adj_points over these particle tiles only (the lists' overflow), or null
    const unsigned* tile_count;
};

// The kernel at delta = x_s - x_b as three numbers: W, gradW = c delta and
// (with HESS) the Hessian c I + e delta delta^T, with c = sigma/h^5 g1(q),
// e = sigma/h^5 g2(q) q / r^2, g1 = f'(q)/q and g2 = d g1/dq
// (kernels/M4_spline.jl:13-36).  r = |delta|, ir = 1/r (0 at r = 0), h and
// invh = 1/h: 1/q = h ir, so no pair needs a division.  The pair terms need
// the Hessian only in products with vectors, H v = c v + e (delta . v) delta,
// so it is never formed.
template <bool HESS>
__device__ __forceinline__ void m4_wce(double r, double ir, double h, double invh, double& W, double& c, double& e) {
    const double q = r * invh;
    const double iq = h * ir;
    const double sig = inv_pi<double>();
    const double ih3 = invh * invh * invh, ih5 = ih3 * invh * invh;
    double f, g1, g2;
    if (q < 1.0) {
        f = 1.0 + q * q * (0.75 * q - 1.5);
        g1 = 2.25 * q - 3.0;
        g2 = 2.25;
    } else {
        const double a = fmax(2.0 - q, 0.0);
        f = 0.25 * a * a * a;
        g1 = -0.75 * a * a * iq;
        g2 = 0.75 * a * (q + 2.0) * (iq * iq);
    }
    W = sig * ih3 * f;
    c = sig * ih5 * g1;
    e = HESS ? sig * ih5 * g2 * q * (ir * ir) : 0.0;  // 0 at r = 0 (ir = 0)
}

// The same for a kernel other than M4 (id k, 3D norm sig): f from kern_fdf,
// g1 = f'(q)/q and g2 = d g1/dq from kern_g12, with 1/q = h ir.
template <bool HESS>
__device__ __forceinline__ void kern_wce(int k, double sig, double r, double ir, double h, double invh, double& W,
                                         double& c, double& e) {
    const double q = r * invh;
    double f, df, g1, g2;
    kern_fdf<double>(k, q, f, df);
    kern_g12(k, q, h * ir, g1, g2);
    const double ih3 = invh * invh * invh, ih5 = ih3 * invh * invh;
    W = sig * ih3 * f;
    c = sig * ih5 * g1;
    e = HESS ? sig * ih5 * g2 * q * (ir * ir) : 0.0;
}

// W, c (and e) of the context's kernel: KF = 0 is the M4 code, KF = 1 any
// other family (the warp-uniform id in pt.kern)
template <int KF, bool HESS>
__device__ __forceinline__ void wce(const TreeView<double>& pt, double r, double ir, double h, double invh, double& W,
                                    double& c, double& e) {
    if constexpr (KF == 0) m4_wce<HESS>(r, ir, h, invh, W, c, e);
    else kern_wce<HESS>(pt.kern, (double)pt.sig, r, ir, h, invh, W, c, e);
}

// Per-particle sums of the pair terms; the particle's factors 1/rho_b,
// m_b/rho_b and m_b are applied once after its last pair:
// dL/dm_b = sW / rho_b + sD, dL/dA_c,b = m_b/rho_b sA_c,
// dL/dx_b = -(m_b/rho_b vS + m_b vD)
// (DG: the catalog has a density gradient; without one sD and vD are 0)
template <int KC, bool DG> struct AdjAcc {
    static constexpr int NF = 4 + KC + (DG ? 4 : 0);  // fields, in the order of f()
    double sW, vS[3], sA[KC], sD, vD[3];
    __device__ __forceinline__ void zero() {
        sW = 0.0; sD = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) { vS[d] = 0.0; vD[d] = 0.0; }
#pragma unroll
        for (int c = 0; c < KC; ++c) sA[c] = 0.0;
    }
    // field i: sW, vS (3), sA (KC), sD, vD (3)
    __device__ __forceinline__ double& f(int i) {
        return i == 0 ? sW : (i < 4 ? vS[i - 1] : (i < 4 + KC ? sA[i - 4] : (i == 4 + KC ? sD : vD[i - 5 - KC])));
    }
};

// The sum cotangents of a pair's sample, by meaning: S1, G (3), Dm, Dg (3),
// Sw_c, Sg_c (3 per column); a scalar catalog (SCAL) has S1 and Sw_c only.
// RowsStrided reads compact row r at ls[r * rs] (rows S1, G, Dm, Dg, Sw_c,
// Sg_c in that order, kc columns; SCAL: S1, Sw_c): the staged rows of
// k_adj_points or the global cotangent rows.
struct RowsStrided {
    const double* ls;
    int64_t rs;
    int kc;
    template <bool SCAL> __device__ __forceinline__ double S1() const { return ls[0]; }
    __device__ __forceinline__ double G(int d) const { return ls[(1 + d) * rs]; }
    __device__ __forceinline__ double Dm() const { return ls[4 * rs]; }
    __device__ __forceinline__ double Dg(int d) const { return ls[(5 + d) * rs]; }
    template <bool SCAL> __device__ __forceinline__ double Sw(int c) const { return ls[((SCAL ? 1 : 8) + c) * rs]; }
    __device__ __forceinline__ double Sg(int c, int d) const { return ls[(8 + kc + 3 * c + d) * rs]; }
};
// Per-sample records of k_adj_bodies: x, y, z, h_a, 1/h_a, then the sum
// cotangents with the columns at fixed places for KC columns (those past the
// catalog's kc are 0), padded to whole 16-byte pairs: one record is read with
// 128-bit loads, where separate arrays would take a 32-byte sector per value.
// Order: S1, G (3, not SCAL), Sw_c, Sg_c (3 per column, not SCAL), then with a
// density gradient Dm, Dg (3).
template <int KC, bool SCAL, bool DG> struct AdjRec {
    static constexpr int SW = SCAL ? 1 : 4, SG = SW + KC, DM = SG + (SCAL ? 0 : 3 * KC);
    static constexpr int NQ = DM + (DG ? 4 : 0);
    static constexpr int N = (5 + NQ + 1) & ~1;  // doubles per record
};
template <int KC, bool SCAL, bool DG> struct RowsRec {
    using RC = AdjRec<KC, SCAL, DG>;
    double q[RC::N];  // the whole record, cotangents from q[5]
    template <bool S> __device__ __forceinline__ double S1() const { return q[5]; }
    __device__ __forceinline__ double G(int d) const { return q[6 + d]; }
    __device__ __forceinline__ double Dm() const { return q[5 + RC::DM]; }
    __device__ __forceinline__ double Dg(int d) const { return q[6 + RC::DM + d]; }
    template <bool S> __device__ __forceinline__ double Sw(int c) const { return q[5 + RC::SW + c]; }
    __device__ __forceinline__ double Sg(int c, int d) const { return q[5 + RC::SG + 3 * c + d]; }
};

// The terms of one pair (sample at (sxv, syv, szv) with h_a = ha, 1/ha = iha;
// particle xb, hb, ihb = 1/hb, columns Ab) with the sample's sum cotangents R.
template <int ST, int KC, bool SCAL, bool DG, int KF, class Rows>
__device__ __forceinline__ void adj_pair(const TreeView<double>& pt, const double xb[3], double hb, double ihb,
                                         const double (&Ab)[KC], int kc, double sxv, double syv, double szv, double ha,
                                         double iha, const Rows& R, AdjAcc<KC, DG>& S) {
    const double dl[3] = {sxv - xb[0], syv - xb[1], szv - xb[2]};
    const double r2 = dl[0] * dl[0] + dl[1] * dl[1] + dl[2] * dl[2];
    const double ir = (r2 > 0.0) ? rsqrt(r2) : 0.0;
    const double r = r2 * ir;
    double W, c, e;
    if (ST == ST_GATHER) {
        wce<KF, !SCAL>(pt, r, ir, ha, iha, W, c, e);
    } else if (ST == ST_SCATTER) {
        wce<KF, !SCAL>(pt, r, ir, hb, ihb, W, c, e);
    } else {
        double Wb, cb, eb;
        wce<KF, !SCAL>(pt, r, ir, ha, iha, W, c, e);
        wce<KF, !SCAL>(pt, r, ir, hb, ihb, Wb, cb, eb);
        W = 0.5 * (W + Wb);
        c = 0.5 * (c + cb);
        e = 0.5 * (e + eb);
    }
    double aS = R.template S1<SCAL>();
    if constexpr (SCAL) {
#pragma unroll
        for (int q = 0; q < KC; ++q) {
            if (q < kc) {
                const double lsw = R.template Sw<SCAL>(q);
                aS += lsw * Ab[q];
                S.sA[q] += lsw * W;
            }
        }
        S.sW += aS * W;
        const double ac = aS * c;
        for (int d = 0; d < 3; ++d) S.vS[d] += ac * dl[d];
        return;
    }
    double aG[3] = {R.G(0), R.G(1), R.G(2)};
#pragma unroll
    for (int q = 0; q < KC; ++q) {
        if (q < kc) {
            const double lsw = R.template Sw<SCAL>(q);
            const double lsg[3] = {R.Sg(q, 0), R.Sg(q, 1), R.Sg(q, 2)};
            aS += lsw * Ab[q];
            aG[0] += Ab[q] * lsg[0]; aG[1] += Ab[q] * lsg[1]; aG[2] += Ab[q] * lsg[2];
            S.sA[q] += lsw * W + c * (lsg[0] * dl[0] + lsg[1] * dl[1] + lsg[2] * dl[2]);
        }
    }
    // v . gradW = c (delta . v), H v = c v + e (delta . v) delta
    const double dG = aG[0] * dl[0] + aG[1] * dl[1] + aG[2] * dl[2];
    S.sW += aS * W + c * dG;
    const double k = aS * c + e * dG;
    for (int d = 0; d < 3; ++d) S.vS[d] += k * dl[d] + c * aG[d];
    if constexpr (DG) {
        const double lDm = R.Dm();
        const double lDg[3] = {R.Dg(0), R.Dg(1), R.Dg(2)};
        const double dD = lDg[0] * dl[0] + lDg[1] * dl[1] + lDg[2] * dl[2];
        S.sD += lDm * W + c * dD;
        const double kd = lDm * c + e * dD;
        for (int d = 0; d < 3; ++d) S.vD[d] += kd * dl[d] + c * lDg[d];
    }
}

// the gradients of particle b (Morton position) from its sums
template <int KC, bool DG>
__device__ __forceinline__ void adj_write(const AdjArgs& A, int64_t b, const AdjAcc<KC, DG>& S, double mb, double rhob,
                                          int kc) {
    const double mr = mb / rhob;
    const int64_t o = A.porder[b];
    A.gm[o] = S.sW / rhob + S.sD;
    A.gx[o] = -(mr * S.vS[0] + mb * S.vD[0]);
    A.gy[o] = -(mr * S.vS[1] + mb * S.vD[1]);
    A.gz[o] = -(mr * S.vS[2] + mb * S.vD[2]);
#pragma unroll
    for (int c = 0; c < KC; ++c)
        if (c < kc && A.gcol[c]) A.gcol[c][o] = mr * S.sA[c];
}

struct AStage {
    double sx[SPAN], sy[SPAN], sz[SPAN], sh[SPAN];  // samples of the span, h_a
    double sih[SPAN];                               // 1 / h_a
    float4 Q[SPAN];   // the samples relative to the warp anchor, float h_a
    float2 AB[SPAN];  // their squared radius thresholds (surely in, maybe in)
    float4 PP[SPAN];  // the warp's particles relative to the warp anchor
    float2 PAB[SPAN]; // their squared radius thresholds
};

// SCAL: every output of the catalog is a (plain or Shepard) scalar, so only
// lambda_S1 and lambda_Sw_c can be non-zero: the pair terms drop the Hessian
// and the gradient cotangents (the same values as the general form, which
// adds exact zeros).
// A pair reads 8 + 4 kc sum cotangents of its sample (1 + kc for scalar
// catalogs: lambda_S1 and lambda_Sw_c).  Every particle of the warp that pairs
// with a sample reads the same ones, so they are staged in shared memory once
// per span, one coalesced load per row.  The general form stages up to 4
// columns (24 rows of 32 doubles per warp); with 8 it would pass the 48 KB of
// static shared memory of a block and reads them from global memory instead.
template <int KC, bool SCAL> struct ALam {
    double q[(SCAL ? 1 + KC : 8 + 4 * KC) * SPAN];  // staged row r of span sample j at r * SPAN + j
};
// the cotangent row (in A.lam) of staged row r
template <bool SCAL> __device__ __forceinline__ int lam_row(int r) { return SCAL ? (r == 0 ? 0 : 7 + r) : r; }

// COL: the pair-list pass of the two-kernel path (the list form): the same
// walk and pair decisions, with each lane's accepted samples of a span
// written to its tile's chain of list blocks instead of summed.
template <int ST, int KC, bool SCAL, int KF, bool COL = false>
__global__ void __launch_bounds__(128, (COL || SCAL) ? 8 : 4) k_adj_points(const AdjArgs A) {
    __shared__ AStage stage_all[4];
    constexpr bool STAGE = !COL && (SCAL || KC <= 4);
    __shared__ ALam<STAGE ? KC : 1, SCAL> lam_all[STAGE ? 4 : 1];
    const TreeView<double>& pt = A.pt;
    const TreeView<double>& sv = A.sv;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    AStage& st = stage_all[wib];
    int64_t tile = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    if (A.tile_list) {  // the tiles the two-kernel path handed back
        if (tile >= (int64_t)*A.tile_count) return;
        tile = A.tile_list[tile];
    }
    if (tile * 32 >= pt.n) return;  // warp-uniform
    const int64_t b = tile * 32 + lane;
    const bool valid = b < pt.n;
    double xb[3] = {0.0, 0.0, 0.0}, hb = 0.0, mb = 0.0, rhob = 1.0, Ab[KC];
#pragma unroll
    for (int c = 0; c < KC; ++c) Ab[c] = 0.0;
    if (valid) {
        xb[0] = pt.x[b]; xb[1] = pt.y[b]; xb[2] = pt.z[b];
        hb = pt.h[b]; mb = pt.m[b]; rhob = pt.rho[b];
#pragma unroll
        for (int c = 0; c < KC; ++c)
            if (c < A.kc) Ab[c] = A.colT[c][b];
    }
    // the support K (2 for M4) in double and float, and the float margin of
    // K h: 2 h is exact in float, K h in general one rounding away
    const double Kd = (KF == 0) ? 2.0 : pt.Kd;
    const float Kf = (KF == 0) ? 2.f : pt.Kf;
    const float km = (KF == 0) ? 2.f * U1 : 3.f * U1;
    // this particle's own support radius^2, with the forward's operation order
    const double rb = X<double>::mul(Kd, hb);
    const double rb2 = X<double>::mul(rb, rb);
    // float pair tests against a band (as in the forward's float walk): the
    // particle relative to the warp anchor (the first valid particle) with its
    // rounding error, its radius bounds and the warp-wide maxima of both
    const unsigned vmask = __ballot_sync(PSB_FULL, valid);
    const int first = vmask ? __ffs(vmask) - 1 : 0;
    const double cw[3] = {__shfl_sync(PSB_FULL, xb[0], first), __shfl_sync(PSB_FULL, xb[1], first),
                          __shfl_sync(PSB_FULL, xb[2], first)};
    const float P[3] = {(float)(xb[0] - cw[0]), (float)(xb[1] - cw[1]), (float)(xb[2] - cw[2])};
    float esmax = U1 * (fabsf(P[0]) + fabsf(P[1]) + fabsf(P[2])) + 1e-30f;
    float rblo = 0.f, rbmax = 0.f;
    if (ST != ST_GATHER) {
        rblo = __double2float_rd(rb) * (1.f - 2.f * U1);
        rbmax = __double2float_ru(rb) * (1.f + 2.f * U1);
    }
    const float rbhi = rbmax;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        esmax = fmaxf(esmax, __shfl_xor_sync(PSB_FULL, esmax, o));
        rbmax = fmaxf(rbmax, __shfl_xor_sync(PSB_FULL, rbmax, o));
    }
    const double ihb = 1.0 / hb;
    AdjAcc<KC, !SCAL> S;
    S.zero();
    const int kc = A.kc;
    const int64_t L = A.lam_stride;
    unsigned long long n_pairs = 0, n_spans = 0, n_parts = 0, n_leaves = 0;  // work counters (warp-uniform)
    int64_t steps = 0;

    const double* lst = lam_all[STAGE ? wib : 0].q;  // the span's staged cotangents
    // li: the sample; jj: its slot in the span
    auto pair = [&](int64_t li, int jj, double sxv, double syv, double szv, double ha, double iha) {
        ++n_pairs;
        // row r of this sample: staged, or from global memory
        const RowsStrided R{STAGE ? lst + jj : A.lam + li, STAGE ? (int64_t)SPAN : L, kc};
        adj_pair<ST, KC, SCAL, !SCAL, KF>(pt, xb, hb, ihb, Ab, kc, sxv, syv, szv, ha, iha, R, S);
    };

    // COL: this tile's chain of list blocks (block, this lane's entries in it)
    int64_t blk = -1;
    int pos = 0;
    bool dead = false;  // the pool ran out: the tile is listed for k_adj_points
    auto emit = [&](int64_t lo, unsigned acc) {
        const bool want = acc != 0;
        if (dead || !__any_sync(PSB_FULL, want)) return;
        if (blk < 0 || __any_sync(PSB_FULL, want && pos == ADJ_CH)) {  // a new block for the warp
            unsigned long long nb = 0;
            if (lane == 0) nb = atomicAdd(A.al.top, 1u);
            nb = __shfl_sync(PSB_FULL, nb, 0);
            if ((int64_t)nb >= A.al.nblocks) {
                dead = true;
                return;
            }
            if (blk >= 0) {
                A.al.bcnt[blk * 32 + lane] = (uint8_t)pos;
                if (lane == 0) A.al.bnext[blk] = (int32_t)nb;
            } else if (lane == 0) {
                A.al.head[tile] = (int32_t)nb;
            }
            if (lane == 0) A.al.btile[nb] = (int32_t)tile;
            blk = (int64_t)nb;
            pos = 0;
        }
        if (want) {
            A.al.ent[((size_t)blk * ADJ_CH + pos) * 32 + lane] = make_uint2((unsigned)lo, acc);
            ++pos;
        }
    };

    // node test seen from the particle, on the float node records (box
    // rounded outwards, scale = max h_a rounded up): the largest sample radius
    // in the node for gather, the particle's own for scatter, the larger for
    // symmetric.  A lower bound of the distance against an upper bound of
    // the radius never prunes a node holding a pair (the pair test itself
    // stays exact).
    const float pf[3] = {(float)xb[0], (float)xb[1], (float)xb[2]};
    const float pem = U1 * fmaxf(fmaxf(fabsf(pf[0]), fabsf(pf[1])), fabsf(pf[2])) + 1e-30f;
    const float rb2_hi = __double2float_ru(rb2) * (1.f + RELM);
    constexpr int SN = (ST == ST_GATHER) ? ST_SCATTER : ((ST == ST_SCATTER) ? ST_GATHER : ST_SYMMETRIC);
    auto node_fn = [&](int ni) -> bool {
        const float4 lo = __ldg(&sv.node_lo[ni]), hi = __ldg(&sv.node_hi[ni]);
        return !(lb_d2_pbox(pf, pem, lo, hi) > hi_r2_node<SN>(rb2_hi, lo.w, Kf));
    };
    auto span_fn = [&](int64_t lo, int cnt, bool part) {
        const unsigned parts = __ballot_sync(PSB_FULL, part);
        if (!parts) return;
        ++n_spans;
        n_parts += __popc(parts);
        n_leaves += cnt;
        // one error bound E for every float distance of the span (the
        // samples are stored relative to the span's first sample)
        const float o0 = (float)(__ldg(&sv.x[lo]) - cw[0]);
        const float o1 = (float)(__ldg(&sv.y[lo]) - cw[1]);
        const float o2 = (float)(__ldg(&sv.z[lo]) - cw[2]);
        const float2 sb = __ldg(&sv.spanb[lo]);
        const float eqm = U1 * (2.f * sb.x + 2.f * (fabsf(o0) + fabsf(o1) + fabsf(o2))) * (1.f + 4.f * U1);
        float rmax = rbmax;
        if (ST != ST_SCATTER) rmax = fmaxf(rmax, Kf * sb.y * (1.f + km));
        const float E = 1.7320508f * (esmax + eqm) + 4.f * U1 * rmax + 1e-30f;
        // squared radius thresholds of this lane's particle and of sample
        // `lane` (surely in: d2 < A; maybe in: d2 <= B)
        float As = 0.f, Bs = 0.f, Aj = 0.f, Bj = 0.f;
        if (ST != ST_GATHER) {  // the particle's own radius K h_b
            const float il = fmaxf((rblo - E) * (1.f - 4.f * U1), 0.f), ih = (rbhi + E) * (1.f + 4.f * U1);
            As = il * il;
            Bs = ih * ih;
        }
        float4 Qme = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        if (lane < cnt) {
            st.sx[lane] = __ldg(&sv.x[lo + lane]); st.sy[lane] = __ldg(&sv.y[lo + lane]);
            st.sz[lane] = __ldg(&sv.z[lo + lane]); st.sh[lane] = __ldg(&sv.h[lo + lane]);
            if (!COL) st.sih[lane] = 1.0 / st.sh[lane];
            const float4 Lq = __ldg(&sv.leaf4[lo + lane]);
            Qme = make_float4(Lq.x + o0, Lq.y + o1, Lq.z + o2, Lq.w);
            st.Q[lane] = Qme;
            if (ST != ST_SCATTER) {  // the sample's radius K h_a
                const float rahi = Kf * Lq.w * (1.f + km), ralo = Kf * Lq.w * (1.f - km);
                const float il = fmaxf((ralo - E) * (1.f - 4.f * U1), 0.f), ih = (rahi + E) * (1.f + 4.f * U1);
                Aj = il * il;
                Bj = ih * ih;
                st.AB[lane] = make_float2(Aj, Bj);
            }
        }
        const int np = __popc(parts);
        const bool by_particle = 3 * np >= 2 * cnt;  // warp-uniform
        if (!by_particle) {
            st.PP[lane] = make_float4(P[0], P[1], P[2], 0.f);
            st.PAB[lane] = make_float2(As, Bs);
        }
        __syncwarp();
        unsigned acc = 0, maybe = 0;
        if (!by_particle) {
            // few particles take part: sample `lane` against each of them
            for (unsigned pp = parts; pp; pp &= pp - 1) {
                const int s = __ffs(pp) - 1;
                const float4 Pp = st.PP[s];
                const float2 ab = st.PAB[s];
                const float dx = Pp.x - Qme.x, dy = Pp.y - Qme.y, dz = Pp.z - Qme.z;
                const float d2 = dx * dx + dy * dy + dz * dz;
                const float At = (ST == ST_GATHER) ? Aj : ((ST == ST_SCATTER) ? ab.x : fmaxf(ab.x, Aj));
                const float Bt = (ST == ST_GATHER) ? Bj : ((ST == ST_SCATTER) ? ab.y : fmaxf(ab.y, Bj));
                const unsigned bi = __ballot_sync(PSB_FULL, lane < cnt && d2 < At);
                const unsigned bm = __ballot_sync(PSB_FULL, lane < cnt && d2 <= Bt);
                if (lane == s) { acc = bi; maybe = bm; }
            }
        } else if (part) {
            // this lane's particle against every sample of the span
#pragma unroll 4
            for (int j = 0; j < cnt; ++j) {
                const float4 Q = st.Q[j];
                const float dx = P[0] - Q.x, dy = P[1] - Q.y, dz = P[2] - Q.z;
                const float d2 = dx * dx + dy * dy + dz * dz;
                float At = As, Bt = Bs;
                if (ST != ST_SCATTER) {
                    const float2 ab = st.AB[j];
                    At = (ST == ST_GATHER) ? ab.x : fmaxf(As, ab.x);
                    Bt = (ST == ST_GATHER) ? ab.y : fmaxf(Bs, ab.y);
                }
                acc |= (unsigned)(d2 < At) << j;
                maybe |= (unsigned)(d2 <= Bt) << j;
            }
        }
        // undecided pairs: the forward's exact test
        for (unsigned u = maybe & ~acc; u; u &= u - 1) {
            const int jj = __ffs(u) - 1;
            const double ps[3] = {st.sx[jj], st.sy[jj], st.sz[jj]};
            const double ra = X<double>::mul(Kd, st.sh[jj]);
            const double ra2 = X<double>::mul(ra, ra);
            const double e2 = ex_d2_pp<double>(ps, xb[0], xb[1], xb[2]);
            if (e2 <= ex_r2<ST, double>(ra2, hb, Kd)) acc |= 1u << jj;
        }
        if constexpr (COL) {
            emit(lo, acc);
        } else {
            if constexpr (STAGE) {  // stage the span's cotangent rows (a warp-uniform decision)
                if (__any_sync(PSB_FULL, acc != 0)) {
                    double* lw = lam_all[wib].q;
                    const int nq = SCAL ? 1 + kc : 8 + 4 * kc;
                    if (lane < cnt)
                        for (int r = 0; r < nq; ++r)
                            lw[r * SPAN + lane] = __ldg(&A.lam[lam_row<SCAL>(r) * L + lo + lane]);
                    __syncwarp();
                }
            }
            for (; acc; acc &= acc - 1) {
                const int jj = __ffs(acc) - 1;
                pair(lo + jj, jj, st.sx[jj], st.sy[jj], st.sz[jj], st.sh[jj], st.sih[jj]);
            }
            if constexpr (STAGE) __syncwarp();  // the rows are read before the next span's
        }
    };
    const int32_t start = (sv.root == 0) ? (int32_t)sv.n : sv.root;
    const bool ok = warp_traverse_spans(start, sv.n, sv.links, sv.escape, valid, node_fn, span_fn, steps);

    if constexpr (COL) {
        if (dead) {
            if (lane == 0) {
                A.al.head[tile] = -2;
                A.al.ovf_tiles[atomicAdd(A.al.ovf_count, 1u)] = (int32_t)tile;
            }
        } else if (blk >= 0) {
            A.al.bcnt[blk * 32 + lane] = (uint8_t)pos;
            if (lane == 0) A.al.bnext[blk] = -1;
        } else if (lane == 0) {
            A.al.head[tile] = -1;
        }
    } else if (valid) {
        adj_write<KC, !SCAL>(A, b, S, mb, rhob, kc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_pairs += __shfl_xor_sync(PSB_FULL, n_pairs, o);
    if (lane == 0 && A.stats) {
        atomicAdd(&A.stats[0], n_pairs);
        atomicAdd(&A.stats[2], (unsigned long long)steps);
        atomicAdd(&A.stats[3], n_spans);
        atomicAdd(&A.stats[4], n_parts);
        atomicAdd(&A.stats[5], n_leaves);
    }

    if (!ok && lane == 0) atomicOr(A.err, PSB_DERR_TRAVERSAL);
}

// The pair terms of the two-kernel path, one list block per warp.  A block
// holds at most ADJ_CH entries for each of its tile's 32 particles, so the work
// items are of like size however long a particle's list is; but within one
// the particles' pairs are few or many (one particle per lane kept 12 of 32
// lanes busy).  So the block's pairs, particle after particle, are dealt out
// in 32 equal runs: a lane sums its run particle by particle, writes what it
// holds alone, and leaves what it shares with its neighbours (its first and
// last particle) in shared memory, where each particle's shares are then added
// in the order of the lanes.  Runs and order follow from the block alone.
// Each pair reads its sample as one record (AdjRec) with 128-bit loads.
// Bound by FP64 issue and the records' L1 traffic: 2M Plummer particles,
// 128^3 grid, 8 fields: 10.1 -> 5.4 ms.  CTAs of one warp, 16 per SM (4 of four: 6.0 ms, a CTA lasts as
// long as its longest warp; 20 at fewer registers: slower).
constexpr int ADJ_BODY_THREADS = 32, ADJ_BODY_CTAS = 16;
template <int ST, int KC, bool SCAL, bool DG, int KF>
__global__ void __launch_bounds__(ADJ_BODY_THREADS, ADJ_BODY_CTAS) k_adj_bodies(const __grid_constant__ AdjArgs A) {
    using Acc = AdjAcc<KC, DG>;
    using RC = AdjRec<KC, SCAL, DG>;
    struct Stage {
        double pd[5 + KC][32];          // particles: x, y, z, h, 1/h, columns
        double seg[2][Acc::NF][32];     // a lane's first and last particle
        int off[33];                    // pairs before each particle
    };
    __shared__ Stage stage_all[ADJ_BODY_THREADS / 32];
    const TreeView<double>& pt = A.pt;
    const int lane = threadIdx.x & 31;
    Stage& st = stage_all[threadIdx.x >> 5];
    const int64_t blk = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int64_t used = (int64_t)*A.al.top;
    if (blk >= (used < A.al.nblocks ? used : A.al.nblocks)) return;  // warp-uniform
    const int64_t tile = A.al.btile[blk];
    // A tile the pool ran out on is k_adj_points' (its last block's counts
    // were never written): skip its blocks.
    const int32_t head = A.al.head[tile];
    if (head == -2) return;  // warp-uniform
    // a tile's only block holds its particles' sums (k_adj_combine starts from
    // the first block's sums, so both give the same bits)
    const bool single = head == blk && A.al.bnext[blk] < 0;
    const int kc = A.kc;
    const uint2* ent = A.al.ent + (size_t)blk * ADJ_CH * 32;
    int cnt = 0;  // pairs of particle `lane` in the block
    {
        const int64_t b = tile * 32 + lane;
        const bool valid = b < pt.n;
        const double hb = valid ? pt.h[b] : 1.0;
        st.pd[0][lane] = valid ? pt.x[b] : 0.0;
        st.pd[1][lane] = valid ? pt.y[b] : 0.0;
        st.pd[2][lane] = valid ? pt.z[b] : 0.0;
        st.pd[3][lane] = hb;
        st.pd[4][lane] = 1.0 / hb;
#pragma unroll
        for (int c = 0; c < KC; ++c) st.pd[5 + c][lane] = (valid && c < kc) ? A.colT[c][b] : 0.0;
        const int ne = valid ? A.al.bcnt[blk * 32 + lane] : 0;
        for (int e = 0; e < ne; ++e) cnt += __popc(ent[e * 32 + lane].y);
        int s = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(PSB_FULL, s, o);
            if (lane >= o) s += t;
        }
        st.off[lane + 1] = s;
        if (lane == 0) st.off[0] = 0;
    }
    __syncwarp();
    const int P = st.off[32];
    auto emit = [&](int q, Acc& S) {  // the block's sums of particle q
        if (single) {
            const int64_t b = tile * 32 + q;
            if (b < pt.n) adj_write<KC, DG>(A, b, S, pt.m[b], pt.rho[b], kc);
        } else {
            double* o = A.al.part + (size_t)blk * Acc::NF * 32 + q;
#pragma unroll
            for (int f = 0; f < Acc::NF; ++f) o[(size_t)f * 32] = S.f(f);
        }
    };
    Acc S;
    S.zero();
    {
        const int i0 = P * lane / 32, i1 = P * (lane + 1) / 32;  // this lane's run
        if (i0 < i1) {
            int p = 0;  // the particle of pair i0: the last one with off[p] <= i0
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                if (st.off[p + o] <= i0) p += o;
            double xb[3], hb, ihb, Ab[KC];
            auto load = [&]() {
                xb[0] = st.pd[0][p]; xb[1] = st.pd[1][p]; xb[2] = st.pd[2][p];
                hb = st.pd[3][p]; ihb = st.pd[4][p];
#pragma unroll
                for (int c = 0; c < KC; ++c) Ab[c] = st.pd[5 + c][p];
            };
            load();
            int skip = i0 - st.off[p], e = 0, end = st.off[p + 1];
            uint2 q = ent[p];
            while (skip >= __popc(q.y)) {
                skip -= __popc(q.y);
                ++e;
                q = ent[e * 32 + p];
            }
            for (; skip > 0; --skip) q.y &= q.y - 1;
            bool first = true;  // the lane's first particle
            for (int i = i0; i < i1; ++i) {
                const double2* rp = reinterpret_cast<const double2*>(
                    A.lamT + (int64_t)(q.x + (unsigned)__ffs(q.y) - 1u) * RC::N);
                q.y &= q.y - 1;
                RowsRec<KC, SCAL, DG> R;
#pragma unroll
                for (int k = 0; k < RC::N / 2; ++k) {
                    const double2 v = __ldg(rp + k);
                    R.q[2 * k] = v.x;
                    R.q[2 * k + 1] = v.y;
                }
                adj_pair<ST, KC, SCAL, DG, KF>(pt, xb, hb, ihb, Ab, kc, R.q[0], R.q[1], R.q[2], R.q[3], R.q[4], R, S);
                if (i + 1 == end) {  // the particle's last pair
                    if (first) {
#pragma unroll
                        for (int f = 0; f < Acc::NF; ++f) st.seg[0][f][lane] = S.f(f);
                    } else {
                        emit(p, S);
                    }
                    first = false;
                    S.zero();
                    if (i + 1 < i1) {
                        do ++p;
                        while (st.off[p + 1] == end);
                        end = st.off[p + 1];
                        load();
                        e = 0;
                        q = ent[p];
                    }
                } else if (q.y == 0) {
                    ++e;
                    q = ent[e * 32 + p];
                }
            }
            if (i1 != end) {  // the particle goes on in the next lane
#pragma unroll
                for (int f = 0; f < Acc::NF; ++f) st.seg[first ? 0 : 1][f][lane] = S.f(f);
            }
        }
    }
    __syncwarp();
    // lane q: particle q, unless one lane held all of it and more before it
    const int o0 = st.off[lane], o1 = st.off[lane + 1];
    if (o1 > o0) {
        const int a = (32 * (o0 + 1) + P - 1) / P - 1, b = (32 * o1 + P - 1) / P - 1;  // lanes of its first and last pair
        const bool mid = P * a / 32 < o0;  // lane a began with another particle
        if (!(a == b && mid)) {
#pragma unroll
            for (int f = 0; f < Acc::NF; ++f) S.f(f) = st.seg[mid ? 1 : 0][f][a];
            for (int l = a + 1; l <= b; ++l) {
                if (P * l / 32 == P * (l + 1) / 32) continue;
#pragma unroll
                for (int f = 0; f < Acc::NF; ++f) S.f(f) += st.seg[0][f][l];
            }
            emit(lane, S);
        }
    } else {
        S.zero();
        emit(lane, S);
    }
    if (lane == 0 && A.stats) atomicAdd(&A.stats[6], (unsigned long long)P);
}

// The gradients of each particle of a tile of several blocks (and zeros for
// a tile without pairs): its blocks' partial sums added in the order of its
// tile's chain (the order the walk met the spans), then the particle's
// factors (adj_write).  The blocks' boundaries follow from the
// walk, so the result does not depend on the pool or on which block landed
// where in it.
template <int KC, bool DG>
__global__ void __launch_bounds__(128) k_adj_combine(const __grid_constant__ AdjArgs A) {
    using Acc = AdjAcc<KC, DG>;
    const TreeView<double>& pt = A.pt;
    const int lane = threadIdx.x & 31;
    const int64_t tile = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (tile * 32 >= pt.n) return;
    const int64_t b = tile * 32 + lane;
    if (b >= pt.n) return;
    int64_t blk = A.al.head[tile];
    if (blk == -2) return;  // overflowed: k_adj_points owns the tile
    Acc T;
    T.zero();
    if (blk >= 0) {
        int64_t nxt = A.al.bnext[blk];
        if (nxt < 0) return;  // one block: k_adj_bodies wrote the gradients
        const double* o = A.al.part + (size_t)blk * Acc::NF * 32 + lane;
#pragma unroll
        for (int f = 0; f < Acc::NF; ++f) T.f(f) = o[(size_t)f * 32];
        for (blk = nxt; blk >= 0; blk = A.al.bnext[blk]) {
            o = A.al.part + (size_t)blk * Acc::NF * 32 + lane;
#pragma unroll
            for (int f = 0; f < Acc::NF; ++f) T.f(f) += o[(size_t)f * 32];
        }
    }
    adj_write<KC, DG>(A, b, T, pt.m[b], pt.rho[b], A.kc);
}

// The records of k_adj_bodies (AdjRec), one per sample of the sample tree:
// position, h_a, 1/h_a and the sum cotangents (lam: rows [q][sample] in the
// tree's order) at the record's fixed places.
template <int KC, bool SCAL, bool DG>
__global__ void k_adj_rows(const double* lam, int64_t ns, int kc, const TreeView<double> sv, double* rec) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    using RC = AdjRec<KC, SCAL, DG>;
    double v[RC::N];
    const double h = sv.h[i];
#pragma unroll
    for (int r = 0; r < RC::N; ++r) v[r] = 0.0;
    v[0] = sv.x[i]; v[1] = sv.y[i]; v[2] = sv.z[i]; v[3] = h; v[4] = 1.0 / h;
    auto row = [&](int r) { return lam[(int64_t)r * ns + i]; };  // compact row r (kc columns)
    v[5] = row(0);
#pragma unroll
    for (int c = 0; c < KC; ++c) {
        if (c >= kc) continue;
        v[5 + RC::SW + c] = row(8 + c);
        if (!SCAL)
            for (int d = 0; d < 3; ++d) v[5 + RC::SG + 3 * c + d] = row(8 + kc + 3 * c + d);
    }
    if (!SCAL)
        for (int d = 0; d < 3; ++d) v[6 + d] = row(1 + d);
    if (DG)
        for (int d = 0; d < 4; ++d) v[5 + RC::DM + d] = row(4 + d);
    double2* o = reinterpret_cast<double2*>(rec + i * RC::N);
#pragma unroll
    for (int r = 0; r < RC::N / 2; ++r) o[r] = make_double2(v[2 * r], v[2 * r + 1]);
}

// line-integrated kernel and its r-derivative: the slope of the table segment
// that line_W interpolates on (LUT_N entries over [0, K], K the support,
// idq = 1/spacing)
__device__ __forceinline__ void line_Wd(double r, double invh, const double* lut, double K, double idq, double& W,
                                        double& dW) {
    const double q = r * invh;
    if (q >= K) { W = 0.0; dW = 0.0; return; }
    const double idxf = q * idq + 1.0;
    int i = (int)idxf;
    i = i < 1 ? 1 : (i > LUT_N - 1 ? LUT_N - 1 : i);
    const double t = idxf - (double)i;
    const double l0 = __ldg(&lut[i - 1]), l1 = __ldg(&lut[i]);
    W = invh * (l0 * (1.0 - t) + l1 * t);
    dW = invh * invh * (l1 - l0) * idq;
}

// A particle of the beam adjoint and the pixels its support can reach.
template <int KC> struct BeamPart {
    double x[3], h, ih, mr;
    double A[KC];
    double u, w, ru, rw;   // centre and half widths on the frame plane, in pixels
    int i0, i1, j0, j1;    // pixels inside those (empty: i1 < i0 or j1 < j0)
};
// Partial gradients: sum aS W, sum s (D - (D.m) m), sum lambda_Sw_c W
template <int KC> struct BeamAcc {
    double m, x[3], A[KC];
    __device__ __forceinline__ void zero() {
        m = 0.0;
        for (int d = 0; d < 3; ++d) x[d] = 0.0;
#pragma unroll
        for (int c = 0; c < KC; ++c) A[c] = 0.0;
    }
    __device__ __forceinline__ void add_xor(int o) {
        m += __shfl_xor_sync(PSB_FULL, m, o);
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] += __shfl_xor_sync(PSB_FULL, x[d], o);
#pragma unroll
        for (int c = 0; c < KC; ++c) A[c] += __shfl_xor_sync(PSB_FULL, A[c], o);
    }
};

// One warp per 32 particles.  A particle's pixels are those of the bounding
// rectangle of its support on the frame plane, re-decided with the forward's
// line distance.  A particle of at most BEAM_LANE pixels is one lane's; up to
// BEAM_GROUP eight lanes share it (4 x 2 pixels at a time, four particles
// side by side), larger ones the warp (8 x 4).  One thread per particle kept
// 17 of 32 lanes active (supports span decades in pixels), visited a pixel
// more than needed on every side, and divided four times a pair: 1M clump
// particles, 512^2 beam: 10.0 -> 3.1 ms.
constexpr int BEAM_LANE = 12, BEAM_GROUP = 160;
template <int ST, int KC>
__global__ void __launch_bounds__(128, 4) k_adj_beam(const __grid_constant__ AdjArgs A) {
    const TreeView<double>& pt = A.pt;
    const int lane = threadIdx.x & 31;
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b - lane >= pt.n) return;  // warp-uniform
    const bool valid = b < pt.n;
    const int kc = A.kc;
    const SampleSrc<double>& B = A.beam;
    const double* f = B.frame;
    const double K = pt.Kd;  // the support (2 for M4)
    const double idq = (double)(LUT_N - 1) / K;
    const double dxi = X<double>::div(X<double>::sub(B.params[1], B.params[0]), (double)(B.nx - 1));
    const double deta = X<double>::div(X<double>::sub(B.params[3], B.params[2]), (double)(B.ny - 1));
    const int64_t L = A.lam_stride;
    unsigned n_pairs = 0;

    BeamPart<KC> P;
    P.i0 = P.j0 = 0;
    P.i1 = P.j1 = -1;
    if (valid) {
        P.x[0] = pt.x[b]; P.x[1] = pt.y[b]; P.x[2] = pt.z[b];
        P.h = pt.h[b];
        P.ih = 1.0 / P.h;
        P.mr = pt.m[b] / pt.rho[b];
#pragma unroll
        for (int c = 0; c < KC; ++c) P.A[c] = (c < kc) ? A.colT[c][b] : 0.0;
        // the particle on the frame plane (frame axes orthonormal), in pixels
        const double v[3] = {P.x[0] - f[0], P.x[1] - f[1], P.x[2] - f[2]};
        const double R = K * fmax(fabs(P.h), A.ha_max);
        P.u = (v[0] * f[3] + v[1] * f[4] + v[2] * f[5] - B.params[0]) / dxi;
        P.w = (v[0] * f[6] + v[1] * f[7] + v[2] * f[8] - B.params[2]) / deta;
        // a frame orthonormal to 1e-9 and the roundings of the projection
        const double slack = 1e-7 * (fabs(v[0]) + fabs(v[1]) + fabs(v[2]) + R);
        P.ru = (R + slack) / fabs(dxi);
        P.rw = (R + slack) / fabs(deta);
        auto range = [](double c, double r, int64_t n, int& a, int& z) {
            const double lo = ceil(c - r), hi = floor(c + r);
            a = lo > 0.0 ? (lo < (double)n ? (int)lo : (int)n) : 0;
            z = hi < (double)(n - 1) ? (hi >= 0.0 ? (int)hi : -1) : (int)(n - 1);
        };
        if (P.u == P.u && P.w == P.w && P.ru == P.ru && P.rw == P.rw) {
            range(P.u, P.ru, B.nx, P.i0, P.i1);
            range(P.w, P.rw, B.ny, P.j0, P.j1);
        }
    }
    // pixel (i, j) of particle q
    auto pixel = [&](const BeamPart<KC>& q, BeamAcc<KC>& S, int i, int j) {
        // the forward's sample coordinates (sample_coords) and line distance
        const double xi = X<double>::add(B.params[0], X<double>::mul((double)i, dxi));
        const double eta = X<double>::add(B.params[2], X<double>::mul((double)j, deta));
        double o[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
            o[c] = X<double>::add(X<double>::add(f[c], X<double>::mul(xi, f[3 + c])), X<double>::mul(eta, f[6 + c]));
        const double* m = f + 9;
        const int64_t k = i + B.nx * (int64_t)j;
        double ha = 0.0;
        if (ST != ST_SCATTER) ha = (A.hmode == PSB_H_PER_SAMPLE) ? A.hs[k] : A.hs[0];
        const double ra = X<double>::mul(K, ha);
        const double e2 = ex_d2_line<double>(o, m, q.x[0], q.x[1], q.x[2]);
        if (!(e2 <= ex_r2<ST, double>(X<double>::mul(ra, ra), q.h, K))) return;
        ++n_pairs;
        const double ir = e2 > 0.0 ? rsqrt(e2) : 0.0;
        const double dr = e2 > 0.0 ? e2 * ir : 0.0;
        double W, dW;
        if (ST == ST_GATHER) {
            line_Wd(dr, 1.0 / ha, A.lut, K, idq, W, dW);
        } else if (ST == ST_SCATTER) {
            line_Wd(dr, q.ih, A.lut, K, idq, W, dW);
        } else {
            double Wb, db;
            line_Wd(dr, 1.0 / ha, A.lut, K, idq, W, dW);
            line_Wd(dr, q.ih, A.lut, K, idq, Wb, db);
            W = 0.5 * (W + Wb);
            dW = 0.5 * (dW + db);
        }
        double aS = __ldg(&A.lam[k]);
#pragma unroll
        for (int c = 0; c < KC; ++c) {
            if (c < kc) {
                const double lsw = __ldg(&A.lam[(1 + c) * L + k]);
                aS += lsw * q.A[c];
                S.A[c] += lsw * W;
            }
        }
        S.m += aS * W;
        // d r_perp / d x_b = (D - (D.m) m) / r_perp, D = x_b - o (0 at r_perp = 0: ir = 0)
        const double D[3] = {q.x[0] - o[0], q.x[1] - o[1], q.x[2] - o[2]};
        const double Dm = D[0] * m[0] + D[1] * m[1] + D[2] * m[2];
        const double s = aS * dW * ir;
#pragma unroll
        for (int d = 0; d < 3; ++d) S.x[d] += s * (D[d] - Dm * m[d]);
    };
    auto write = [&](int64_t q, const BeamAcc<KC>& S, double mr) {
        const int64_t ob = A.porder[q];
        A.gm[ob] = S.m / pt.rho[q];
        A.gx[ob] = mr * S.x[0]; A.gy[ob] = mr * S.x[1]; A.gz[ob] = mr * S.x[2];
#pragma unroll
        for (int c = 0; c < KC; ++c)
            if (c < kc && A.gcol[c]) A.gcol[c][ob] = mr * S.A[c];
    };
    const int64_t npix = valid ? (int64_t)max(P.i1 - P.i0 + 1, 0) * max(P.j1 - P.j0 + 1, 0) : 0;
    BeamAcc<KC> S;
    S.zero();
    if (valid && npix <= BEAM_LANE) {
        for (int j = P.j0; j <= P.j1; ++j)
            for (int i = P.i0; i <= P.i1; ++i) pixel(P, S, i, j);
        write(b, S, P.mr);
    }
    // particle `from` of the warp, in every lane of a group
    auto fetch = [&](int from) -> BeamPart<KC> {
        BeamPart<KC> q;
#pragma unroll
        for (int d = 0; d < 3; ++d) q.x[d] = __shfl_sync(PSB_FULL, P.x[d], from);
        q.h = __shfl_sync(PSB_FULL, P.h, from);
        q.ih = __shfl_sync(PSB_FULL, P.ih, from);
        q.mr = __shfl_sync(PSB_FULL, P.mr, from);
#pragma unroll
        for (int c = 0; c < KC; ++c) q.A[c] = __shfl_sync(PSB_FULL, P.A[c], from);
        q.u = __shfl_sync(PSB_FULL, P.u, from);
        q.w = __shfl_sync(PSB_FULL, P.w, from);
        q.ru = __shfl_sync(PSB_FULL, P.ru, from);
        q.rw = __shfl_sync(PSB_FULL, P.rw, from);
        q.i0 = __shfl_sync(PSB_FULL, P.i0, from);
        q.i1 = __shfl_sync(PSB_FULL, P.i1, from);
        q.j0 = __shfl_sync(PSB_FULL, P.j0, from);
        q.j1 = __shfl_sync(PSB_FULL, P.j1, from);
        return q;
    };
    // the pixels of row j inside the support's ellipse
    auto row = [&](const BeamPart<KC>& q, int j, int& a, int& z) {
        const double t = ((double)j - q.w) / q.rw, c = q.ru * sqrt(fmax(1.0 - t * t, 0.0)) + 1e-6;
        a = max(q.i0, (int)fmax(ceil(q.u - c), -1.0));
        z = min(q.i1, (int)fmin(floor(q.u + c), 2147483000.0));
    };
    unsigned todo = __ballot_sync(PSB_FULL, valid && npix > BEAM_LANE && npix <= BEAM_GROUP);
    while (todo) {  // eight lanes per particle, four particles at a time
        const int g = lane >> 3;
        unsigned t = todo;
        for (int k = 0; k < g; ++k) t &= t - 1;
        const int from = t ? __ffs(t) - 1 : 0;
        const BeamPart<KC> q = fetch(from);
        S.zero();
        if (t)
            for (int j = q.j0 + ((lane >> 2) & 1); j <= q.j1; j += 2)
                for (int i = q.i0 + (lane & 3); i <= q.i1; i += 4) pixel(q, S, i, j);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) S.add_xor(o);
        if (t && (lane & 7) == 0) write(b - lane + from, S, q.mr);
        for (int k = 0; k < 4; ++k) todo &= todo - 1;
    }
    for (todo = __ballot_sync(PSB_FULL, valid && npix > BEAM_GROUP); todo; todo &= todo - 1) {  // the whole warp
        const int from = __ffs(todo) - 1;
        const BeamPart<KC> q = fetch(from);
        S.zero();
        for (int j = q.j0 + (lane >> 3); j <= q.j1; j += 4) {
            int a, z;
            row(q, j, a, z);
            for (int i = a + (lane & 7); i <= z; i += 8) pixel(q, S, i, j);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) S.add_xor(o);
        if (lane == 0) write(b - lane + from, S, q.mr);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_pairs += __shfl_xor_sync(PSB_FULL, n_pairs, o);
    if (lane == 0 && A.stats && n_pairs) atomicAdd(&A.stats[0], (unsigned long long)n_pairs);
}

// sample coordinates of every sample of a source (grid, box) as arrays
__global__ void k_sample_xyz(const SampleSrc<double> S, int64_t ns, double* x, double* y, double* z) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ns) return;
    double p[3], d[3];
    sample_coords(S, k, p, d);
    x[k] = p[0]; y[k] = p[1]; z[k] = p[2];
}

// lam_out[q][i] = lam_in[q][order[i]]: sum cotangents in the sample tree's order
__global__ void k_gather_rows(const double* in, const int64_t* order, int64_t n, int nq, double* out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t s = order[i];
    for (int q = 0; q < nq; ++q) out[q * n + i] = in[q * n + s];
}

}  // namespace psb
