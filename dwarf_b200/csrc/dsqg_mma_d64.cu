// Tensor-core kernels, D = 64 with the usual dense window (instantiated apart: the kernels take minutes to compile).
#include "dsqg_mma_kernels.cuh"

namespace dsqg {

cudaError_t launch_fwd_mma_d64(const FwdArgs& a, const Taps& t, cudaStream_t s) {
    return fwd_launch_mma<64, 32>(a, t, s);
}

cudaError_t launch_bwd_mma_d64(const BwdArgs& a, const Taps& t, cudaStream_t s, int stages) {
    return bwd_launch_mma<64, 32>(a, t, s, stages);
}

}  // namespace dsqg
