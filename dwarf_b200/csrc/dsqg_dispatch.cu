// Chooses between the tensor-core kernels (bf16; D in {32, 64} with or without scale_embed,
// D in {48, 80, 96, 128} without) and the generic CUDA-core kernels (everything else: fp32 storage,
// other head sizes, dense windows wider than the tensor-core kernels are built for).  One
// decision per call, made on the host from the shape alone.
#include <atomic>
#include <mutex>

#include "dsqg_common.cuh"

namespace dsqg {

// 0 = automatic, 1 = always the generic kernels, 2 = the register-fed tensor-core kernels (what the
// automatic choice uses where they apply, except for the one case in umma_pays()), 3 = the forward with TMA-staged V wherever it applies
// (dsqg_staged.cu; not chosen automatically: it measures slower on B200), 4 = the forward with the
// dense window on tcgen05 / tensor memory wherever it applies (dsqg_umma.cu; chosen automatically in the case of umma_pays() only).
static std::atomic<int> g_path{0};
constexpr int kErrorDevices = 64;

// Where the tcgen05 forward is taken instead of the register-fed one: 128-byte rows (D = 64), no sparse taps, at least two
// 128-row tiles for each SM's persistent block.  The line was drawn when the register-fed kernel took 56.1 us at 3,072 tiles (tcgen05 49).  It no longer
// stands for speed: the register-fed kernel is 8 to 15 % ahead at every size now (offsets 0..31, L2 cold, tcgen05 / register-fed: 6,144 tiles (16x12x4096)
// 85.0 / 78.8 us, 3,072 tiles 50.2 / 46.1, 1,536 tiles 31.7 / 27.6, 768 tiles 21.5 / 19.5, 320 tiles 15.4 / 13.3).  Moving it changes which kernel's bits
// these calls return (dsqg_b200.h says which), and that is all that keeps it.
static bool umma_pays(const FwdArgs& a, const Taps& t, int dtype) {
    return a.D == 64 && t.n_sparse == 0 && !a.strided &&
           (long long)a.B * a.H * ((a.N + 127) / 128) >= 2 * 148 && umma_supported(dtype, a.D, t, a.scale_embed != nullptr);
}

cudaError_t launch_fwd(const FwdArgs& a, const Taps& t, int dtype, cudaStream_t s) {
    const int path = g_path.load();
    if (path == 0 && umma_pays(a, t, dtype)) return launch_fwd_umma(a, t, s);
    if (path == 4 && !a.strided && umma_supported(dtype, a.D, t, a.scale_embed != nullptr)) return launch_fwd_umma(a, t, s);
    if (path == 3 && staged_supported(dtype, a.D, t, a.scale_embed != nullptr)) return launch_fwd_staged(a, t, s);
    if (path != 1 && (mma_fwd_supported(dtype, a.D, t, a.scale_embed != nullptr) || mma_tail_supported(dtype, a.D, t, a.scale_embed != nullptr)))
        return launch_fwd_mma(a, t, s);
    return launch_fwd_generic(a, t, dtype, s);
}

cudaError_t launch_bwd(const BwdArgs& a, const Taps& t, int dtype, cudaStream_t s, int stages) {
    const int path = g_path.load();
    if (path != 1 && (mma_path_supported(dtype, a.D, t, a.scale_embed != nullptr) || mma_tail_supported(dtype, a.D, t, a.scale_embed != nullptr)))
        return launch_bwd_mma(a, t, s, stages);
    return launch_bwd_generic(a, t, dtype, s, stages);
}

// One page of page-locked host memory, asked for once (also while a stream is being captured: no stream takes part in it).
static int* error_words() {
    static std::mutex mu;
    static int* words = nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!words) {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        void* p = nullptr;
        if (cudaHostAlloc(&p, kErrorDevices * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
            words = static_cast<int*>(p);
            for (int i = 0; i < kErrorDevices; ++i) words[i] = 0;
        } else {
            cudaGetLastError();
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
    return words;
}
static int* host_word() {
    int dev = 0;
    int* words = error_words();
    return words && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kErrorDevices ? words + dev : nullptr;
}
int* wait_error_word() {
    void* p = nullptr;
    int* w = host_word();
    return w && cudaHostGetDevicePointer(&p, w, 0) == cudaSuccess ? static_cast<int*>(p) : nullptr;
}
int wait_error_seen() {
    const volatile int* w = host_word();
    return w ? *w : 0;
}
static void clear_wait_error() {
    volatile int* w = host_word();
    if (w) *w = 0;
}

}  // namespace dsqg

extern "C" int dsqg_set_kernel_path(int path) {
    if (path < 0 || path > 4) return DSQG_ERR_UNSUPPORTED;
    dsqg::g_path.store(path);
    return DSQG_OK;
}

extern "C" int dsqg_device_error(int reset) {
    int v = 0, w = 0, g = 0;
    if (cudaDeviceSynchronize() != cudaSuccess) { cudaGetLastError(); return -1; }
    if (dsqg::read_stage_error(&v, reset != 0) != cudaSuccess) return -1;
    if (dsqg::read_umma_error(&w, reset != 0) != cudaSuccess) return -1;
    if (dsqg::read_wgrad_error(&g, reset != 0) != cudaSuccess) return -1;
    if (reset) dsqg::clear_wait_error();
    return v ? v : w ? w : g;
}

extern "C" int dsqg_test_wait_timeout(long long limit_cycles, void* stream) {
    if (limit_cycles < 1 || limit_cycles > 2000000000LL) return DSQG_ERR_UNSUPPORTED;
    return dsqg::launch_wait_timeout(limit_cycles, 0x7e57, static_cast<cudaStream_t>(stream)) == cudaSuccess ? DSQG_OK : DSQG_ERR_CUDA;
}
