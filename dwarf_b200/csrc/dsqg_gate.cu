// Backward of the sigmoid gate that dsqg_fwd_strided folds into its epilogue.
//
// The forward wrote y = o * sigmoid(gate), o being the DSQG output (DWARF
// train/train_2048_condU.py:184-191: `out * torch.sigmoid(self.gate_proj(x))`).  Given dy this
// kernel forms, in one pass over the three tensors,
//   dout  = dy * sigmoid(gate)                    the gradient the DSQG backward consumes,
//   dgate = dy * o * s (1 - s) = dy * y * (1 - s) the gradient of the gate projection's output,
//   delta = sum_d dout * o = sum_d dy * y         per (batch, head, row): what the DSQG backward
//                                                 otherwise derives from its saved output,
// so the un-gated output o never has to be stored.  bf16 tensors, fp32 arithmetic.
#include "dsqg_common.cuh"

namespace dsqg {
namespace {

// LPR lanes per (batch, row, head), eight elements each.  Five tensors pass through once, so memory is the bound: with
// one thread per row (the row's 16-byte pieces 64 bytes or more apart from lane to lane) a warp's load touched 16 lines
// for 512 bytes; B32 H8 N2048 D32 (168 MB) 46.7 us then, 28.8 us now.  The packed backward does the same inside its dQ kernel (gate_row).
//
// Up to D = 32 delta is summed element by element, lane after lane, as one thread would: ds = P (dP - delta) is rounded to bf16, and another order
// moves single roundings, which a gradient that nearly cancels (a bias on every key) shows.  At 40 registers (six CTAs per SM)
// the chain hides behind the loads: 28.9 us with it and without (31.0 with five CTAs).  At D = 64 and 128 it would not: 24.7 against 22.8 us
// (B8 H12 N2048) and 35.6 against 28.8 (B8 H8); there the lanes' sums are added in pairs.
template <int LPR>
__global__ void __launch_bounds__(256, 6)
gate_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ y,
                const __nv_bfloat16* __restrict__ gate, __nv_bfloat16* __restrict__ dgate, __nv_bfloat16* __restrict__ dout, const dsqg_strides st,
                float* __restrict__ delta, int B, int H, int N, int D) {
    stream_wait();
    const unsigned row = (blockIdx.x * 256u + threadIdx.x) / LPR, c = threadIdx.x % LPR * 8;
    if (row >= (unsigned)B * N * H) return;                    // whole lane groups leave
    const unsigned h = row % H, bn = row / H, n = bn % N, b = bn / N;
    const size_t at = (size_t)b * st.batch + (size_t)h * st.head + (size_t)n * st.row + c;
    float d[8] = {}, o[8] = {};
    if (c < D) {
        float g[8], go[8], gg[8];
        load8(gate + at, g); load8(dy + at, d); load8(y + at, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float s = __fdividef(1.f, 1.f + __expf(-g[i]));
            go[i] = d[i] * s;
            gg[i] = d[i] * o[i] * (1.f - s);
        }
        store8(dout + at, go); store8(dgate + at, gg);
    }
    const unsigned group = LPR == 32 ? 0xffffffffu : ((1u << LPR) - 1) << ((threadIdx.x & 31) / LPR * LPR);
    float acc = 0.f;
    if constexpr (LPR <= 4) {
#pragma unroll
        for (int l = 0; l < LPR; ++l) {                        // every lane adds its products to what the lane before has; the l-th lane's count
            float t = l ? __shfl_sync(group, acc, l - 1, LPR) : 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) t = fmaf(d[i], o[i], t);
            acc = t;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc = fmaf(d[i], o[i], acc);
#pragma unroll
        for (int l = LPR / 2; l > 0; l >>= 1) acc += __shfl_xor_sync(group, acc, l);
    }
    if (threadIdx.x % LPR == LPR - 1) delta[((size_t)b * H + h) * N + n] = acc;
}

template <int LPR>
cudaError_t gate_launch(const void* dy, const void* y, const void* gate, void* dgate, void* dout, const dsqg_strides& st, float* delta, int B, int H, int N, int D,
                        cudaStream_t s) {
    const long long threads = (long long)B * N * H * LPR;
    return launch_after(gate_bwd_kernel<LPR>, (unsigned)((threads + 255) / 256), 256, 0, s, static_cast<const __nv_bfloat16*>(dy),
                        static_cast<const __nv_bfloat16*>(y), static_cast<const __nv_bfloat16*>(gate), static_cast<__nv_bfloat16*>(dgate),
                        static_cast<__nv_bfloat16*>(dout), st, delta, B, H, N, D);
}

}  // namespace

cudaError_t launch_gate_bwd(const void* dy, const void* y, const void* gate, void* dgate, void* dout, const dsqg_strides& st, float* delta, int B, int H, int N, int D,
                            cudaStream_t s) {
    auto launch = D <= 8 ? gate_launch<1> : D <= 16 ? gate_launch<2> : D <= 32 ? gate_launch<4> : D <= 64 ? gate_launch<8> : gate_launch<16>;
    return launch(dy, y, gate, dgate, dout, st, delta, B, H, N, D, s);
}

}  // namespace dsqg
