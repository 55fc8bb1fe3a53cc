// Tensor-core kernels, D = 32 and 64 with dense windows of more than 33 offsets (instantiated apart: the kernels take minutes to compile).
#include "dsqg_mma_kernels.cuh"

namespace dsqg {

cudaError_t launch_fwd_mma_window(const FwdArgs& a, const Taps& t, cudaStream_t s) {
    if (a.D == 32 && band_width(t) == 48) return fwd_launch_mma<32, 48>(a, t, s);
    if (a.D == 32) return fwd_launch_mma<32, 64>(a, t, s);
    if (band_width(t) == 48) return fwd_launch_mma<64, 48>(a, t, s);
    return fwd_launch_mma<64, 64>(a, t, s);
}

cudaError_t launch_bwd_mma_window(const BwdArgs& a, const Taps& t, cudaStream_t s, int stages) {
    if (a.D == 32 && band_width(t) == 48) return bwd_launch_mma<32, 48>(a, t, s, stages);
    if (a.D == 32) return bwd_launch_mma<32, 64>(a, t, s, stages);
    if (band_width(t) == 48) return bwd_launch_mma<64, 48>(a, t, s, stages);
    return bwd_launch_mma<64, 64>(a, t, s, stages);
}

}  // namespace dsqg
