// Instantiations of the line kernels and the launch front ends.
#include "launch.hpp"
namespace psb {
cudaError_t launch_points_d0(const Args<double>&, int, int, int, cudaStream_t);
cudaError_t launch_points_d1(const Args<double>&, int, int, int, cudaStream_t);
cudaError_t launch_points_f0(const Args<float>&, int, int, int, cudaStream_t);
cudaError_t launch_points_f1(const Args<float>&, int, int, int, cudaStream_t);

template <> cudaError_t launch_points<double>(const Args<double>& a, int prec, int st, int kc, int what, cudaStream_t s) {
    return prec == PREC_FP64 ? launch_points_d0(a, st, kc, what, s) : launch_points_d1(a, st, kc, what, s);
}
template <> cudaError_t launch_points<float>(const Args<float>& a, int prec, int st, int kc, int what, cudaStream_t s) {
    return prec == PREC_FP64 ? launch_points_f0(a, st, kc, what, s) : launch_points_f1(a, st, kc, what, s);
}
template <> cudaError_t launch_lines<double>(const Args<double>& a, int prec, int st, int kc, int what, cudaStream_t s) {
    return prec == PREC_FP64 ? dispatch_lines_p<double, PREC_FP64>(a, st, kc, what, s)
                             : dispatch_lines_p<double, PREC_FP32C>(a, st, kc, what, s);
}
template <> cudaError_t launch_lines<float>(const Args<float>& a, int prec, int st, int kc, int what, cudaStream_t s) {
    return prec == PREC_FP64 ? dispatch_lines_p<float, PREC_FP64>(a, st, kc, what, s)
                             : dispatch_lines_p<float, PREC_FP32C>(a, st, kc, what, s);
}
// defined in inst_line_tile_*.cu
cudaError_t launch_line_tile_d0(const Args<double>&, int, int, bool, cudaStream_t);
cudaError_t launch_line_tile_d1(const Args<double>&, int, int, bool, cudaStream_t);
cudaError_t launch_line_tile(const Args<double>& a, int prec, int st, int kc, bool wide, cudaStream_t s) {
    return prec == PREC_FP64 ? launch_line_tile_d0(a, st, kc, wide, s) : launch_line_tile_d1(a, st, kc, wide, s);
}
cudaError_t launch_line_share(const Args<double>& a, int prec, int st, const int32_t* parent, unsigned* together,
                              cudaStream_t s) {
    const bool d = prec == PREC_FP64;
    auto kern = st == ST_GATHER ? k_line_share<ST_GATHER> : (st == ST_SCATTER ? k_line_share<ST_SCATTER> : k_line_share<ST_SYMMETRIC>);
    kern<<<1, SHARE_THREADS, 0, s>>>(a, parent, d ? LINE_SHARE_FP64 : LINE_SHARE_FP32C,
                                     d ? LINE_SHARE_TILES_FP64 : LINE_SHARE_TILES_FP32C, together);
    return cudaGetLastError();
}
cudaError_t launch_line_warp(const Args<double>& a, int prec, int st, cudaStream_t s) {
    return prec == PREC_FP64 ? dispatch_line_warp<PREC_FP64>(a, st, s) : dispatch_line_warp<PREC_FP32C>(a, st, s);
}
}  // namespace psb
