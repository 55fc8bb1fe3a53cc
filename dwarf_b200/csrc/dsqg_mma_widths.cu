// Tensor-core kernels, the other head widths (instantiated apart: the kernels take minutes to compile).
#include "dsqg_mma_kernels.cuh"

namespace dsqg {

cudaError_t launch_fwd_mma_widths(const FwdArgs& a, const Taps& t, cudaStream_t s) {
    if (a.D == 48) return fwd_launch_mma<48, 32>(a, t, s);
    if (a.D == 80) return fwd_launch_mma<80, 32>(a, t, s);
    if (a.D == 96) return fwd_launch_mma<96, 32>(a, t, s);
    return fwd_launch_mma<128, 32>(a, t, s);
}

cudaError_t launch_bwd_mma_widths(const BwdArgs& a, const Taps& t, cudaStream_t s, int stages) {
    if (a.D == 48) return bwd_launch_mma<48, 32>(a, t, s, stages);
    if (a.D == 80) return bwd_launch_mma<80, 32>(a, t, s, stages);
    if (a.D == 96) return bwd_launch_mma<96, 32>(a, t, s, stages);
    return bwd_launch_mma<128, 32>(a, t, s, stages);
}

}  // namespace dsqg
