// Instantiations of the line tile kernel, PREC_FP64.
#include "launch.hpp"
namespace psb {
cudaError_t launch_line_tile_d0(const Args<double>& a, int st, int kc, bool wide, cudaStream_t s) {
    return dispatch_line_tile<PREC_FP64>(a, st, kc, wide, s);
}
}  // namespace psb
