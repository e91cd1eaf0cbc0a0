// Instantiations of the two-kernel point path: double inputs, PREC_FP32C.
#include "launch.hpp"

namespace psb {
cudaError_t launch_split_d1(const Args<double>& a, int st, int kc, int pass, cudaStream_t s) {
    return dispatch_split_p<double, PREC_FP32C>(a, st, kc, pass, s);
}
}  // namespace psb
