// Tensor-core kernels: what they take, the choice between the instantiations, and those for D = 32.
#include "dsqg_mma_kernels.cuh"

namespace dsqg {

cudaError_t launch_fwd_mma_d64(const FwdArgs& a, const Taps& t, cudaStream_t s);
cudaError_t launch_bwd_mma_d64(const BwdArgs& a, const Taps& t, cudaStream_t s, int stages);
cudaError_t launch_fwd_mma_window(const FwdArgs& a, const Taps& t, cudaStream_t s);
cudaError_t launch_bwd_mma_window(const BwdArgs& a, const Taps& t, cudaStream_t s, int stages);
cudaError_t launch_fwd_mma_widths(const FwdArgs& a, const Taps& t, cudaStream_t s);
cudaError_t launch_bwd_mma_widths(const BwdArgs& a, const Taps& t, cudaStream_t s, int stages);

static bool mma_shape_supported(int dtype, int D, const Taps& t) {
    const int wb = band_width(t);
    return dtype == DSQG_DTYPE_BF16 && (((D == 32 || D == 64) && wb != 0) || ((D == 96 || D == 128) && wb == 32));
}
// Widths with a 16-element tail run on their own kernels when nothing else is asked of them (contiguous tensors, no
// scale_embed); a caller may also pad them, so mma_fwd_supported / mma_path_supported leave them out.
bool mma_tail_supported(int dtype, int D, const Taps& t, bool has_scale_embed) {
    return dtype == DSQG_DTYPE_BF16 && (D == 48 || D == 80) && band_width(t) == 32 && !has_scale_embed;
}
bool mma_fwd_supported(int dtype, int D, const Taps& t, bool has_scale_embed) {
    return mma_shape_supported(dtype, D, t) && (!has_scale_embed || D <= 64);
}
bool mma_path_supported(int dtype, int D, const Taps& t, bool has_scale_embed) {
    return mma_shape_supported(dtype, D, t) && (!has_scale_embed || D <= 64);
}

cudaError_t launch_fwd_mma(const FwdArgs& a, const Taps& t, cudaStream_t s) {
    if (a.D != 32 && a.D != 64) return launch_fwd_mma_widths(a, t, s);
    if (band_width(t) != 32) return launch_fwd_mma_window(a, t, s);
    return a.D == 32 ? fwd_launch_mma<32, 32>(a, t, s) : launch_fwd_mma_d64(a, t, s);
}

cudaError_t launch_bwd_mma(const BwdArgs& a, const Taps& t, cudaStream_t s, int stages) {
    if (a.D != 32 && a.D != 64) return launch_bwd_mma_widths(a, t, s, stages);
    if (band_width(t) != 32) return launch_bwd_mma_window(a, t, s, stages);
    return a.D == 32 ? bwd_launch_mma<32, 32>(a, t, s, stages) : launch_bwd_mma_d64(a, t, s, stages);
}

}  // namespace dsqg
