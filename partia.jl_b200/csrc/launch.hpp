// launch.hpp -- template dispatch of the interpolation kernels.  The
// instantiations are split over inst_*.cu so that they compile in parallel.
#pragma once

#include <algorithm>

#include "k_line_warp.cuh"

namespace psb {

// KF: 0 = the M4 kernel's own code, 1 = the other kernel families (digests
// evaluate no kernel)
template <class T, int P, int S, int W, int KF>
static void dispatch_points_kf(const Args<T>& a, int kc, unsigned g, cudaStream_t s) {
    if constexpr (W != WHAT_INTERP) {
        k_points<T, P, S, 1, W, KF><<<g, 128, 0, s>>>(a);
    } else {
        if (kc <= 1) k_points<T, P, S, 1, W, KF><<<g, 128, 0, s>>>(a);
        else if (kc <= 2) k_points<T, P, S, 2, W, KF><<<g, 128, 0, s>>>(a);
        else if (kc <= 4) k_points<T, P, S, 4, W, KF><<<g, 128, 0, s>>>(a);
        else k_points<T, P, S, 8, W, KF><<<g, 128, 0, s>>>(a);
    }
}
template <class T, int P, int S, int W>
static void dispatch_points_k(const Args<T>& a, int kc, unsigned g, cudaStream_t s) {
    if (W == WHAT_DIGEST || a.tv.kern == KERN_M4) dispatch_points_kf<T, P, S, W, 0>(a, kc, g, s);
    else if constexpr (W != WHAT_DIGEST) dispatch_points_kf<T, P, S, W, 1>(a, kc, g, s);
}

template <class T, int P, int W>
static void dispatch_points_s(const Args<T>& a, int st, int kc, unsigned g, cudaStream_t s) {
    if (st == ST_GATHER) dispatch_points_k<T, P, ST_GATHER, W>(a, kc, g, s);
    else if (st == ST_SCATTER) dispatch_points_k<T, P, ST_SCATTER, W>(a, kc, g, s);
    else dispatch_points_k<T, P, ST_SYMMETRIC, W>(a, kc, g, s);
}

template <class T, int P>
static cudaError_t dispatch_points_p(const Args<T>& a, int st, int kc, int what, cudaStream_t s) {
    unsigned g = (unsigned)((a.src.ntiles + 3) / 4);
    if (g == 0) return cudaSuccess;
    if (what == WHAT_INTERP) dispatch_points_s<T, P, WHAT_INTERP>(a, st, kc, g, s);
    else if (what == WHAT_DENSITY) dispatch_points_s<T, P, WHAT_DENSITY>(a, st, kc, g, s);
    else dispatch_points_s<T, P, WHAT_DIGEST>(a, st, kc, g, s);
    return cudaGetLastError();
}

template <class T, int P, int S, int W>
static void dispatch_lines_k(const Args<T>& a, int kc, unsigned g, size_t smem, cudaStream_t s) {
    if constexpr (W != WHAT_INTERP) {
        k_lines<T, P, S, 1, W><<<g, 128, smem, s>>>(a);
    } else {
        if (kc <= 1) k_lines<T, P, S, 1, W><<<g, 128, smem, s>>>(a);
        else if (kc <= 4) k_lines<T, P, S, 4, W><<<g, 128, smem, s>>>(a);
        else k_lines<T, P, S, 8, W><<<g, 128, smem, s>>>(a);
    }
}

template <class T, int P, int W>
static void dispatch_lines_s(const Args<T>& a, int st, int kc, unsigned g, size_t smem, cudaStream_t s) {
    if (st == ST_GATHER) dispatch_lines_k<T, P, ST_GATHER, W>(a, kc, g, smem, s);
    else if (st == ST_SCATTER) dispatch_lines_k<T, P, ST_SCATTER, W>(a, kc, g, smem, s);
    else dispatch_lines_k<T, P, ST_SYMMETRIC, W>(a, kc, g, smem, s);
}

template <class T, int P>
static cudaError_t dispatch_lines_p(const Args<T>& a, int st, int kc, int what, cudaStream_t s) {
    unsigned g = (unsigned)((a.src.ntiles + 3) / 4);
    if (g == 0) return cudaSuccess;
    // shared memory only for the FP64 sums over the short float table (k_lines)
    size_t smem = (P == PREC_FP64 && a.lut_n == LUT_SHORT_N) ? (size_t)LUT_SHORT_N * sizeof(double) : 0;
    if (what == WHAT_INTERP) dispatch_lines_s<T, P, WHAT_INTERP>(a, st, kc, g, smem, s);
    else dispatch_lines_s<T, P, WHAT_DIGEST>(a, st, kc, g, smem, s);
    return cudaGetLastError();
}

// tiles of lines that run together; wide: eight lanes per line (k_line_tile's G)
template <int P, int S, int G>
static void dispatch_line_tile_s(const Args<double>& a, int kc, cudaStream_t s) {
    const unsigned g = (unsigned)((a.src.ntiles * G + 3) / 4);
    if (kc <= 1) k_line_tile<P, S, 1, G><<<g, 128, 0, s>>>(a);
    else if (kc <= 4) k_line_tile<P, S, 4, G><<<g, 128, 0, s>>>(a);
    else k_line_tile<P, S, 8, G><<<g, 128, 0, s>>>(a);
}
template <int P, int G>
static void dispatch_line_tile_g(const Args<double>& a, int st, int kc, cudaStream_t s) {
    if (st == ST_GATHER) dispatch_line_tile_s<P, ST_GATHER, G>(a, kc, s);
    else if (st == ST_SCATTER) dispatch_line_tile_s<P, ST_SCATTER, G>(a, kc, s);
    else dispatch_line_tile_s<P, ST_SYMMETRIC, G>(a, kc, s);
}
template <int P>
static cudaError_t dispatch_line_tile(const Args<double>& a, int st, int kc, bool wide, cudaStream_t s) {
    if (a.src.ntiles == 0) return cudaSuccess;
    if (wide) dispatch_line_tile_g<P, 8>(a, st, kc, s);
    else dispatch_line_tile_g<P, 1>(a, st, kc, s);
    return cudaGetLastError();
}

// one warp per line: every line, or those of the listed groups
template <int P>
static cudaError_t dispatch_line_warp(const Args<double>& a, int st, cudaStream_t s) {
    const unsigned g = (unsigned)(a.src.ntiles * 8);
    if (g == 0) return cudaSuccess;
    if (st == ST_GATHER) k_line_warp<P, ST_GATHER><<<g, 128, 0, s>>>(a);
    else if (st == ST_SCATTER) k_line_warp<P, ST_SCATTER><<<g, 128, 0, s>>>(a);
    else k_line_warp<P, ST_SYMMETRIC><<<g, 128, 0, s>>>(a);
    return cudaGetLastError();
}

// two-kernel point path over the batch a.sp: the walk (k_collect, then k_heavy for its largest samples), the sums
// over its lists (k_bodies, k_density; first the tiles' blocks,
// then the chunks'), and the fold of the samples with chunks (k_fold)
enum { SPLIT_WALK = 0, SPLIT_FIELDS = 1, SPLIT_DENSITY = 2, SPLIT_FOLD = 3, SPLIT_FOLD_DENSITY = 4, SPLIT_HEAVY = 5 };
template <class T, int P, int S, int KF, bool DG>
static void dispatch_bodies_kfd(const Args<T>& a, int kc, unsigned g, unsigned gc, cudaStream_t s) {
    if (kc <= 1) k_bodies<T, P, S, 1, KF, DG><<<g + gc, BODY_THREADS, 0, s>>>(a, g);
    else if (kc <= 2) k_bodies<T, P, S, 2, KF, DG><<<g + gc, BODY_THREADS, 0, s>>>(a, g);
    else if (kc <= 4) k_bodies<T, P, S, 4, KF, DG><<<g + gc, BODY_THREADS, 0, s>>>(a, g);
    else if (kc == 5) k_bodies<T, P, S, 5, KF, DG><<<g + gc, BODY_THREADS, 0, s>>>(a, g);
    else if (kc <= 6) k_bodies<T, P, S, 6, KF, DG><<<g + gc, BODY_THREADS, 0, s>>>(a, g);
    else k_bodies<T, P, S, 8, KF, DG><<<g + gc, BODY_THREADS, 0, s>>>(a, g);
}
// DG: the catalog has a density gradient (its sums and the masses in
// registers only where they are used)
template <class T, int P, int S, int KF>
static void dispatch_bodies_kf(const Args<T>& a, int kc, unsigned g, unsigned gc, cudaStream_t s) {
    if (a.rec.need_dg) dispatch_bodies_kfd<T, P, S, KF, true>(a, kc, g, gc, s);
    else dispatch_bodies_kfd<T, P, S, KF, false>(a, kc, g, gc, s);
}
template <class T, int P, int S>
static void dispatch_bodies_k(const Args<T>& a, int kc, unsigned g, unsigned gc, cudaStream_t s) {
    if (a.tv.kern == KERN_M4) dispatch_bodies_kf<T, P, S, 0>(a, kc, g, gc, s);
    else dispatch_bodies_kf<T, P, S, 1>(a, kc, g, gc, s);
}

template <class T, int P, int S>
static void dispatch_density_k(const Args<T>& a, unsigned g, unsigned gc, cudaStream_t s) {
    if (a.tv.kern == KERN_M4) k_density<T, P, S, 0><<<g + gc, BODY_THREADS, 0, s>>>(a, g);
    else k_density<T, P, S, 1><<<g + gc, BODY_THREADS, 0, s>>>(a, g);
}

// k_seq: enough warps to fill the GPU, each takes samples until none is left
template <class T, int P, int S>
static void dispatch_seq_s(const Args<T>& a, bool density, cudaStream_t s) {
    const int64_t items = (a.sp.seq_all ? a.sp.ntiles * 32 : 0) + a.sp.ncap;
    const unsigned g = (unsigned)std::min<int64_t>(148 * 8, (items + 3) / 4);
    const bool m4 = a.tv.kern == KERN_M4;
    if (density) {
        if (m4) k_seq<T, P, S, 0, WHAT_DENSITY><<<g, 128, 0, s>>>(a);
        else k_seq<T, P, S, 1, WHAT_DENSITY><<<g, 128, 0, s>>>(a);
    } else {
        if (m4) k_seq<T, P, S, 0, WHAT_INTERP><<<g, 128, 0, s>>>(a);
        else k_seq<T, P, S, 1, WHAT_INTERP><<<g, 128, 0, s>>>(a);
    }
}
template <class T, int P>
static void dispatch_seq(const Args<T>& a, int st, bool density, cudaStream_t s) {
    if (st == ST_GATHER) dispatch_seq_s<T, P, ST_GATHER>(a, density, s);
    else if (st == ST_SCATTER) dispatch_seq_s<T, P, ST_SCATTER>(a, density, s);
    else dispatch_seq_s<T, P, ST_SYMMETRIC>(a, density, s);
}

// the samples of a few parts with a lane each (CHAIN)
template <class T, int P, int S, int KF, bool DG>
static void dispatch_chain_kfd(const Args<T>& a, int kc, unsigned g, cudaStream_t s) {
    if (kc <= 1) k_bodies<T, P, S, 1, KF, DG, true><<<g, BODY_THREADS, 0, s>>>(a, 0);
    else if (kc <= 4) k_bodies<T, P, S, 4, KF, DG, true><<<g, BODY_THREADS, 0, s>>>(a, 0);
    else k_bodies<T, P, S, 8, KF, DG, true><<<g, BODY_THREADS, 0, s>>>(a, 0);
}
template <class T, int P, int S, int KF>
static void dispatch_chain_kf(const Args<T>& a, int kc, bool density, unsigned g, cudaStream_t s) {
    if (density) k_density<T, P, S, KF, true><<<g, BODY_THREADS, 0, s>>>(a, 0);
    else if (a.rec.need_dg) dispatch_chain_kfd<T, P, S, KF, true>(a, kc, g, s);
    else dispatch_chain_kfd<T, P, S, KF, false>(a, kc, g, s);
}
template <class T, int P, int S>
static void dispatch_chain_s(const Args<T>& a, int kc, bool density, unsigned g, cudaStream_t s) {
    if (a.tv.kern == KERN_M4) dispatch_chain_kf<T, P, S, 0>(a, kc, density, g, s);
    else dispatch_chain_kf<T, P, S, 1>(a, kc, density, g, s);
}
template <class T, int P>
static void dispatch_chain(const Args<T>& a, int st, int kc, bool density, cudaStream_t s) {
    const int64_t most = std::min<int64_t>(a.sp.ntiles * 32, a.sp.ncap);
    if (most < (int64_t)CHAIN_SAMPLES) return;
    const unsigned g = (unsigned)((most + BODY_THREADS - 1) / BODY_THREADS);
    if (st == ST_GATHER) dispatch_chain_s<T, P, ST_GATHER>(a, kc, density, g, s);
    else if (st == ST_SCATTER) dispatch_chain_s<T, P, ST_SCATTER>(a, kc, density, g, s);
    else dispatch_chain_s<T, P, ST_SYMMETRIC>(a, kc, density, g, s);
}

template <class T, int P>
static cudaError_t dispatch_split_p(const Args<T>& a, int st, int kc, int pass, cudaStream_t s) {
    // blocks of the tiles' lists and of the chunk pool
    constexpr bool SEQ = sizeof(T) == 8 && P == PREC_FP32C;
    constexpr int BW = BODY_THREADS / 32, WW = WALK_THREADS / 32;
    const unsigned g = (unsigned)((a.sp.ntiles + BW - 1) / BW), gc = SEQ ? 0 : (a.sp.ncap + BODY_THREADS - 1) / BODY_THREADS;
    const unsigned gf = (a.sp.ncap + 127) / 128;
    if (g == 0) return cudaSuccess;
    if (pass == SPLIT_FOLD || pass == SPLIT_FOLD_DENSITY) {
        if constexpr (SEQ) {
            dispatch_seq<T, P>(a, st, pass == SPLIT_FOLD_DENSITY, s);
            if (!a.sp.seq_all) dispatch_chain<T, P>(a, st, kc, pass == SPLIT_FOLD_DENSITY, s);
        } else {
            if (pass == SPLIT_FOLD_DENSITY) k_fold<T, P, 1, WHAT_DENSITY><<<gf, 128, 0, s>>>(a);
            else if (kc <= 1) k_fold<T, P, 1, WHAT_INTERP><<<gf, 128, 0, s>>>(a);
            else if (kc <= 2) k_fold<T, P, 2, WHAT_INTERP><<<gf, 128, 0, s>>>(a);
            else if (kc <= 4) k_fold<T, P, 4, WHAT_INTERP><<<gf, 128, 0, s>>>(a);
            else if (kc == 5) k_fold<T, P, 5, WHAT_INTERP><<<gf, 128, 0, s>>>(a);
            else if (kc <= 6) k_fold<T, P, 6, WHAT_INTERP><<<gf, 128, 0, s>>>(a);
            else k_fold<T, P, 8, WHAT_INTERP><<<gf, 128, 0, s>>>(a);
        }
    } else if (pass == SPLIT_HEAVY) {
        auto kern = st == ST_GATHER ? k_heavy<T, ST_GATHER> : (st == ST_SCATTER ? k_heavy<T, ST_SCATTER> : k_heavy<T, ST_SYMMETRIC>);
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HEAVY_SMEM);
        if (e != cudaSuccess) return e;
        kern<<<std::min(2 * 148u, a.sp.hcap), HEAVY_THREADS, HEAVY_SMEM, s>>>(a);
    } else if (pass == SPLIT_WALK) {
        const unsigned gw = (unsigned)(((a.sp.ntiles << (5 - a.sp.lspt)) + WW - 1) / WW);
        auto walk = [&](auto wide) {
            constexpr bool W = decltype(wide)::value;
            if (st == ST_GATHER) k_collect<T, ST_GATHER, W><<<gw, WALK_THREADS, 0, s>>>(a);
            else if (st == ST_SCATTER) k_collect<T, ST_SCATTER, W><<<gw, WALK_THREADS, 0, s>>>(a);
            else k_collect<T, ST_SYMMETRIC, W><<<gw, WALK_THREADS, 0, s>>>(a);
        };
        if (a.sp.wide) walk(std::true_type());
        else walk(std::false_type());
    } else if (a.sp.seq_all) {  // in FP32C of double particles the fold pass takes all samples
        if constexpr (!SEQ) dispatch_seq<T, P>(a, st, pass == SPLIT_DENSITY, s);
    } else if (pass == SPLIT_DENSITY) {
        if (st == ST_GATHER) dispatch_density_k<T, P, ST_GATHER>(a, g, gc, s);
        else if (st == ST_SCATTER) dispatch_density_k<T, P, ST_SCATTER>(a, g, gc, s);
        else dispatch_density_k<T, P, ST_SYMMETRIC>(a, g, gc, s);
    } else {
        if (st == ST_GATHER) dispatch_bodies_k<T, P, ST_GATHER>(a, kc, g, gc, s);
        else if (st == ST_SCATTER) dispatch_bodies_k<T, P, ST_SCATTER>(a, kc, g, gc, s);
        else dispatch_bodies_k<T, P, ST_SYMMETRIC>(a, kc, g, gc, s);
    }
    return cudaGetLastError();
}

// defined in inst_*.cu
template <class T> cudaError_t launch_points(const Args<T>& a, int prec, int st, int kc, int what, cudaStream_t s);
cudaError_t launch_split_d0(const Args<double>& a, int st, int kc, int pass, cudaStream_t s);
cudaError_t launch_split_d1(const Args<double>& a, int st, int kc, int pass, cudaStream_t s);
cudaError_t launch_split_f0(const Args<float>& a, int st, int kc, int pass, cudaStream_t s);
cudaError_t launch_split_f1(const Args<float>& a, int st, int kc, int pass, cudaStream_t s);
inline cudaError_t launch_split(const Args<double>& a, int prec, int st, int kc, int pass, cudaStream_t s) {
    return prec == PREC_FP64 ? launch_split_d0(a, st, kc, pass, s) : launch_split_d1(a, st, kc, pass, s);
}
inline cudaError_t launch_split(const Args<float>& a, int prec, int st, int kc, int pass, cudaStream_t s) {
    return prec == PREC_FP64 ? launch_split_f0(a, st, kc, pass, s) : launch_split_f1(a, st, kc, pass, s);
}
template <class T> cudaError_t launch_lines(const Args<T>& a, int prec, int st, int kc, int what, cudaStream_t s);
cudaError_t launch_line_tile(const Args<double>& a, int prec, int st, int kc, bool wide, cudaStream_t s);
cudaError_t launch_line_warp(const Args<double>& a, int prec, int st, cudaStream_t s);
cudaError_t launch_line_share(const Args<double>& a, int prec, int st, const int32_t* parent, unsigned* together,
                              cudaStream_t s);

}  // namespace psb
