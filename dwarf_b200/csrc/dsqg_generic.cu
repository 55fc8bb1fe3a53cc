// Generic DSQG kernels: any head dim D = 8k <= 128, any tap set, bf16 or fp32 storage,
// fp32 arithmetic on the CUDA cores.  These are the fp32-I/O instantiation (needed for
// the 1e-5 parity gate against the reference's fp32 PyTorch path) and the fall-back for
// shapes the tensor-core kernels do not cover.  Math follows the DWARF reference kernels
// kernels/dsqg_attention_v3.py:60-163 (forward), :198-275 (dQ, dpos_bias, dscale_embed),
// :282-352 (dK, dV), with the offset set as a runtime argument and the per-head output
// gain of train/train_2048_condU.py:187 fused in.
//
// Mapping of the backward kernels: a group of TPR = next_pow2(D/8) lanes owns one row; every lane holds 8
// contiguous elements of the row in fp32 registers; dot products are reduced with
// xor-shuffles inside the group.  Global loads are 16/32-byte vectors and consecutive
// lanes read consecutive addresses, so each warp touches whole contiguous rows.
#include "dsqg_common.cuh"
#include <type_traits>

namespace dsqg {

namespace {

constexpr int kThreads = 256;
constexpr int kRowsPerBwdTile = 512;   // rows handled by one dQ block (a multiple of every RPB)

template <typename T> struct Exp;
template <> struct Exp<float> { static __device__ __forceinline__ float f(float x) { return expf(x); } };
template <> struct Exp<__nv_bfloat16> { static __device__ __forceinline__ float f(float x) { return __expf(x); } };

// Four elements of a row in fp32.
__device__ __forceinline__ float4 load4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}

// Forward.  LPR lanes hold a row, four elements each; a lane group owns kFwdRows consecutive query rows and
// takes the taps eight at a time (online softmax over the chunks).  What bounds it is the L1 data path, the
// shuffles and issue slots, not the multiply-adds, hence
//   * one 16-byte load of four lanes covers whole 128-byte lines (eight elements per lane, two loads 32 bytes
//     apart, moved the same rows in twice as many passes);
//   * eight consecutive offsets of two consecutive rows touch only nine key rows, loaded once;
//   * the partial dot products of eight taps are summed over the lanes by halving (seven shuffles per row
//     instead of 3 x 8), which leaves one tap's score per lane: its exponential is computed once and handed
//     back with one shuffle;
//   * four taps or less at the end are a chunk of four, and the multiply-adds work on packed pairs.
// fp32, 43 taps, us: B2 H8 N2048 D32 17.5 (19.3 with scalar multiply-adds and chunks of eight only, 31.8 with one row per group and one tap at a
// time; four rows per group or 256 threads 24 and more), B14 97.9 (107.2), B8 H8 N2048 D64 115.0 (122.9), B2 H8 N1500 D128 44.1 (47.0), B1 H8 N300
// D32 5.8 (5.9).  Scores first and values after, the scores waiting in shared memory: 17.6 with 7 CTAs per SM, but 7.4 at B1 H8 N300.
constexpr int kFwdRows = 2, kFwdThreads = 128;

// EXACT: D == 4 LPR, so that the rows of a run are compile-time offsets apart.
template <typename T, int LPR, bool EXACT>
__global__ void __launch_bounds__(kFwdThreads, 4)
fwd_generic_kernel(const FwdArgs a, const Taps t) {
    constexpr int R = kFwdRows, GPB = kFwdThreads / LPR;
    __shared__ float pb_s[DSQG_MAX_TAPS];
    __shared__ int off_s[DSQG_MAX_TAPS];
    stream_wait();
    const int bh = blockIdx.y, h = bh % a.H, N = a.N, D = EXACT ? 4 * LPR : a.D, J = t.J;
    const int g = threadIdx.x / LPR, li = threadIdx.x % LPR, d0 = 4 * li;
    const bool active = d0 < D;
    for (int j = threadIdx.x; j < J; j += kFwdThreads) { pb_s[j] = a.pos_bias[j * a.H + h]; off_s[j] = t.delta(j); }
    __syncthreads();
    const int n0 = (blockIdx.x * GPB + g) * R;
    const size_t base = (size_t)bh * N * D + (active ? d0 : 0);
    const T* kb = static_cast<const T*>(a.k) + base;
    const T* vb = static_cast<const T*>(a.v) + base;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 q[R];
#pragma unroll
    for (int r = 0; r < R; ++r) q[r] = active && n0 + r < N ? load4(static_cast<const T*>(a.q) + base + (size_t)(n0 + r) * D) : zero;
    auto dot = [](const float4& x, const float4& y) {
        const f32x2 s = fma2(pair(x.z, x.w), pair(y.z, y.w), mul2(pair(x.x, x.y), pair(y.x, y.y)));
        float lo, hi;
        unpair(s, lo, hi);
        return lo + hi;
    };
    // Taps j0 .. j0 + C - 1.  RUN: consecutive offsets.  INSIDE: every partner row of the warp exists; otherwise any key row of the
    // sequence stands in for one that does not (its score is -inf), and a value of zero (a weight of 0 would not hold off an infinity or NaN there).
    auto row_at = [&](auto INSIDEC, const T* p, int n, int i) {
        if constexpr (decltype(INSIDEC)::value) return load4(p + (ptrdiff_t)n * D + i * D);
        else return load4(p + (ptrdiff_t)min(max(n + i, 0), N - 1) * D);
    };
    auto scores = [&](auto CC, auto RUNC, auto INSIDEC, int j0, float (&x)[R]) {
        constexpr int C = decltype(CC)::value;
        constexpr bool RUN = decltype(RUNC)::value;
        float part[R][C];
        if constexpr (RUN) {
            const int first = n0 - off_s[j0] - (C - 1);                     // the R + C - 1 rows start here
#pragma unroll
            for (int i = 0; i < R + C - 1; ++i) {
                const float4 k = row_at(INSIDEC, kb, first, i);
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (C - 1 + r - i >= 0 && C - 1 + r - i < C) part[r][C - 1 + r - i] = dot(q[r], k);
            }
        } else {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int dl = off_s[min(j0 + c, J - 1)];
#pragma unroll
                for (int r = 0; r < R; ++r) part[r][c] = dot(q[r], row_at(INSIDEC, kb, n0 - dl, r));
            }
        }
        if (a.scale_embed != nullptr && active) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float4 e = load4(a.scale_embed + (size_t)min(j0 + c, J - 1) * D + d0);
#pragma unroll
                for (int r = 0; r < R; ++r) part[r][c] += dot(q[r], e);
            }
        }
        const int j = j0 + (li & (C - 1)), dl = off_s[min(j, J - 1)];
        const bool mine = j < J && (C == 8 || (li & 7) < C);                // every tap counts on one lane of eight
        const float pb = pb_s[min(j, J - 1)];
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int half = C / 2; half > 0; half >>= 1) {
                const bool up = li & half;
#pragma unroll
                for (int c = 0; c < half; ++c) {
                    const float keep = up ? part[r][c + half] : part[r][c], send = up ? part[r][c] : part[r][c + half];
                    part[r][c] = keep + __shfl_xor_sync(0xffffffffu, send, half);
                }
            }
            float s = part[r][0];
#pragma unroll
            for (int o = C; o < LPR; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            x[r] = mine && n0 + r >= dl ? fmaf(s, a.scale, pb) : -INFINITY;
        }
    };
    f32x2 acc[R][2];
    float m[R], l[R];                       // maximum; sum over this lane's taps only
#pragma unroll
    for (int r = 0; r < R; ++r) { m[r] = -INFINITY; l[r] = 0.f; acc[r][0] = acc[r][1] = 0ull; }
    auto group_max = [](float x) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
        return x;
    };
    auto finite = [](float x) { return x == -INFINITY ? 0.f : x; };
    auto values = [&](auto CC, auto RUNC, auto INSIDEC, int j0, const float (&x)[R]) {
        constexpr int C = decltype(CC)::value;
        constexpr bool RUN = decltype(RUNC)::value, INSIDE = decltype(INSIDEC)::value;
        float p[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            p[r] = Exp<T>::f(x[r] - finite(m[r]));
            l[r] += p[r];
        }
        auto fold = [&](int r, int c, int n, int i, float4 v) {
            if (!INSIDE && (n + i < 0 || n + i >= N)) v = zero;
            const float w = __shfl_sync(0xffffffffu, p[r], c, 8);
            acc[r][0] = fma2(pair(w, w), pair(v.x, v.y), acc[r][0]);
            acc[r][1] = fma2(pair(w, w), pair(v.z, v.w), acc[r][1]);
        };
        if constexpr (RUN) {
            const int first = n0 - off_s[j0] - (C - 1);
#pragma unroll
            for (int i = 0; i < R + C - 1; ++i) {
                const float4 v = row_at(INSIDEC, vb, first, i);
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (C - 1 + r - i >= 0 && C - 1 + r - i < C) fold(r, C - 1 + r - i, first, i, v);
            }
        } else {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int dc = off_s[min(j0 + c, J - 1)];
#pragma unroll
                for (int r = 0; r < R; ++r) fold(r, c, n0 - dc, r, row_at(INSIDEC, vb, n0 - dc, r));
            }
        }
    };
    auto chunk = [&](auto C, auto run, auto inside, int j0) {
        float x[R];
        scores(C, run, inside, j0, x);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float mn = fmaxf(m[r], group_max(x[r])), cor = Exp<T>::f(m[r] - finite(mn));
            m[r] = mn;
            l[r] *= cor;
            acc[r][0] = mul2(acc[r][0], pair(cor, cor)); acc[r][1] = mul2(acc[r][1], pair(cor, cor));
        }
        values(C, run, inside, j0, x);
    };
    using Yes = std::true_type;
    using No = std::false_type;
    std::integral_constant<int, 8> eight;
    std::integral_constant<int, 4> four;
#pragma unroll 1
    for (int j0 = 0; j0 < J; j0 += 8) {
        if (!__any_sync(0xffffffffu, n0 + R - 1 >= off_s[j0])) break;                                // offsets ascend
        const bool run = j0 + 8 <= t.n_dense;
        const bool inside = __all_sync(0xffffffffu, n0 >= off_s[min(j0 + 7, J - 1)] && n0 + R <= N);
        if (j0 + 4 >= J) {
            if (inside) chunk(four, No(), Yes(), j0); else chunk(four, No(), No(), j0);
        } else if (run) {
            if (inside) chunk(eight, Yes(), Yes(), j0); else chunk(eight, Yes(), No(), j0);
        } else {
            if (inside) chunk(eight, No(), Yes(), j0); else chunk(eight, No(), No(), j0);
        }
    }
    const float gain = a.head_gain ? a.head_gain[h] : 1.f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float sum = l[r];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (n0 + r >= N) continue;
        const float inv = sum > 0.f ? gain / sum : 0.f;
        float4 o;
        unpair(acc[r][0], o.x, o.y); unpair(acc[r][1], o.z, o.w);
        if (active)
            store4(static_cast<T*>(a.out) + base + (size_t)(n0 + r) * D, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
        if (li == 0) a.lse[(size_t)bh * N + n0 + r] = sum > 0.f ? m[r] + logf(sum) : -INFINITY;
    }
}

// dQ + row-wise delta + partial sums of dpos_bias / dhead_gain / dscale_embed.
// One block owns kRowsPerBwdTile consecutive rows of one (b,h) and walks them RPB at a time.
// Dynamic shared memory: ds_s[RPB][J] | dg_s[RPB] | (q_s[RPB][D] | dse_acc[J*D] when SE).
template <typename T, int TPR>
__global__ void __launch_bounds__(kThreads)
bwd_dq_generic_kernel(const BwdArgs a, const Taps t) {
    stream_wait();
    constexpr int RPB = kThreads / TPR;
    extern __shared__ float smem[];
    __shared__ float pb_s[DSQG_MAX_TAPS];
    const int J = t.J, D = a.D;
    float* ds_s = smem;                  // [RPB][J]
    float* dg_s = ds_s + RPB * J;        // [RPB]
    float* q_s = dg_s + RPB;             // [RPB][D]
    float* dse_acc = q_s + RPB * D;      // [J*D]
    const bool has_se = a.scale_embed != nullptr;

    const int bh = blockIdx.y, h = bh % a.H;
    const int tile = bh * a.tiles_per_bh + blockIdx.x;
    const int row0 = blockIdx.x * kRowsPerBwdTile;
    const int row_end = min(a.N, row0 + kRowsPerBwdTile);
    const int g = threadIdx.x / TPR, li = threadIdx.x % TPR;
    const int d0 = li * 8;
    const bool active = d0 < D;

    for (int j = threadIdx.x; j < J; j += kThreads) pb_s[j] = a.pos_bias[j * a.H + h];
    if (has_se)
        for (int i = threadIdx.x; i < J * D; i += kThreads) dse_acc[i] = 0.f;
    __syncthreads();

    const size_t base = (size_t)bh * a.N * D;
    const T* qb = static_cast<const T*>(a.q) + base;
    const T* kb = static_cast<const T*>(a.k) + base;
    const T* vb = static_cast<const T*>(a.v) + base;
    const T* ob = static_cast<const T*>(a.out) + base;
    const T* dob = static_cast<const T*>(a.dout) + base;
    T* dqb = static_cast<T*>(a.dq) + base;
    const float gain = a.head_gain ? a.head_gain[h] : 1.f;

    float dpb_r = 0.f;   // thread j < J accumulates dpos_bias[j]
    float dg_r = 0.f;    // thread J accumulates sum_rows dout . o_pre

    for (int r0 = row0; r0 < row_end; r0 += RPB) {
        const int n = r0 + g;
        const bool row_ok = n < row_end;
        float q[8] = {0, 0, 0, 0, 0, 0, 0, 0}, dox[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        float delta = 0.f, lse_n = 0.f;
        if (row_ok && active) {
            float o[8];
            load8(qb + (size_t)n * D + d0, q);
            load8(dob + (size_t)n * D + d0, dox);
            load8(ob + (size_t)n * D + d0, o);
#pragma unroll
            for (int i = 0; i < 8; ++i) delta = fmaf(dox[i], o[i], delta);
        }
        delta = group_sum<TPR>(delta);
        if (row_ok) {
            lse_n = a.lse[(size_t)bh * a.N + n];
            if (li == 0) a.delta[(size_t)bh * a.N + n] = delta;
        }
        float dq[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        float dgrow = 0.f;
        for (int j = 0; j < J; ++j) {
            const int src = n - t.delta(j);
            const bool valid = row_ok && src >= 0;
            float kx[8] = {0, 0, 0, 0, 0, 0, 0, 0}, vx[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (valid && active) {
                load8(kb + (size_t)src * D + d0, kx);
                load8(vb + (size_t)src * D + d0, vx);
                if (has_se) {
                    float se[8];
                    load8(a.scale_embed + (size_t)j * D + d0, se);
#pragma unroll
                    for (int i = 0; i < 8; ++i) kx[i] += se[i];
                }
            }
            float dot_s = 0.f, dot_p = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) { dot_s = fmaf(q[i], kx[i], dot_s); dot_p = fmaf(dox[i], vx[i], dot_p); }
            dot_s = group_sum<TPR>(dot_s);
            dot_p = group_sum<TPR>(dot_p);
            float ds = 0.f;
            if (valid) {
                const float s = dot_s * a.scale + pb_s[j];
                const float p = Exp<T>::f(s - lse_n);
                ds = p * (gain * dot_p - delta);
                dgrow = fmaf(p, dot_p, dgrow);
                const float w = ds * a.scale;
#pragma unroll
                for (int i = 0; i < 8; ++i) dq[i] = fmaf(w, kx[i], dq[i]);
            }
            if (li == 0) ds_s[g * J + j] = ds;
        }
        if (row_ok && active) store8(dqb + (size_t)n * D + d0, dq);
        if (li == 0) dg_s[g] = row_ok ? dgrow : 0.f;
        if (has_se && active) {
#pragma unroll
            for (int i = 0; i < 8; ++i) q_s[g * D + d0 + i] = q[i];   // zeros for rows past the end
        }
        __syncthreads();
        if (threadIdx.x < J) {
            for (int r = 0; r < RPB; ++r) dpb_r += ds_s[r * J + threadIdx.x];
        } else if (threadIdx.x == J) {
            for (int r = 0; r < RPB; ++r) dg_r += dg_s[r];
        }
        if (has_se) {
            for (int idx = threadIdx.x; idx < J * D; idx += kThreads) {
                const int j = idx / D, d = idx - j * D;
                float acc = dse_acc[idx];
                for (int r = 0; r < RPB; ++r) acc = fmaf(ds_s[r * J + j], q_s[r * D + d], acc);
                dse_acc[idx] = acc;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < J) a.dpb_part[(size_t)tile * J + threadIdx.x] = dpb_r;
    else if (threadIdx.x == J) a.dg_part[tile] = dg_r;
    if (has_se)
        for (int idx = threadIdx.x; idx < J * D; idx += kThreads)
            a.dse_part[(size_t)tile * J * D + idx] = dse_acc[idx] * a.scale;
}

// dK, dV: the group owns key row m and visits the query rows m + delta_j that read it.
template <typename T, int TPR>
__global__ void __launch_bounds__(kThreads)
bwd_dkdv_generic_kernel(const BwdArgs a, const Taps t) {
    stream_wait();
    constexpr int RPB = kThreads / TPR;
    __shared__ float pb_s[DSQG_MAX_TAPS];
    const int J = t.J, D = a.D;
    const int bh = blockIdx.y, h = bh % a.H;
    const int g = threadIdx.x / TPR, li = threadIdx.x % TPR;
    const int d0 = li * 8;
    const bool active = d0 < D;
    const int m = blockIdx.x * RPB + g;
    const bool row_ok = m < a.N;
    for (int j = threadIdx.x; j < J; j += kThreads) pb_s[j] = a.pos_bias[j * a.H + h];
    __syncthreads();

    const size_t base = (size_t)bh * a.N * D;
    const T* qb = static_cast<const T*>(a.q) + base;
    const T* dob = static_cast<const T*>(a.dout) + base;
    const float* lse_b = a.lse + (size_t)bh * a.N;
    const float* delta_b = a.delta + (size_t)bh * a.N;
    const float gain = a.head_gain ? a.head_gain[h] : 1.f;
    const bool has_se = a.scale_embed != nullptr;

    float kx[8] = {0, 0, 0, 0, 0, 0, 0, 0}, vx[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (row_ok && active) {
        load8(static_cast<const T*>(a.k) + base + (size_t)m * D + d0, kx);
        load8(static_cast<const T*>(a.v) + base + (size_t)m * D + d0, vx);
    }
    float dk[8] = {0, 0, 0, 0, 0, 0, 0, 0}, dv[8] = {0, 0, 0, 0, 0, 0, 0, 0};

    for (int j = 0; j < J; ++j) {
        const int n = m + t.delta(j);
        const bool valid = row_ok && n < a.N;
        float qx[8] = {0, 0, 0, 0, 0, 0, 0, 0}, dox[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        float kk[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) kk[i] = kx[i];
        if (valid && active) {
            load8(qb + (size_t)n * D + d0, qx);
            load8(dob + (size_t)n * D + d0, dox);
            if (has_se) {
                float se[8];
                load8(a.scale_embed + (size_t)j * D + d0, se);
#pragma unroll
                for (int i = 0; i < 8; ++i) kk[i] += se[i];
            }
        }
        float dot_s = 0.f, dot_p = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) { dot_s = fmaf(qx[i], kk[i], dot_s); dot_p = fmaf(dox[i], vx[i], dot_p); }
        dot_s = group_sum<TPR>(dot_s);
        dot_p = group_sum<TPR>(dot_p);
        if (valid) {
            const float s = dot_s * a.scale + pb_s[j];
            const float p = Exp<T>::f(s - lse_b[n]);
            const float ds = p * (gain * dot_p - delta_b[n]);
            const float wv = p * gain, wk = ds * a.scale;
#pragma unroll
            for (int i = 0; i < 8; ++i) { dv[i] = fmaf(wv, dox[i], dv[i]); dk[i] = fmaf(wk, qx[i], dk[i]); }
        }
    }
    if (row_ok && active) {
        store8(static_cast<T*>(a.dk) + base + (size_t)m * D + d0, dk);
        store8(static_cast<T*>(a.dv) + base + (size_t)m * D + d0, dv);
    }
}

}  // namespace

// One block per output element; the partials are summed in a fixed order (per-thread strided
// partial sums, then a fixed shared-memory tree), so the result is bitwise reproducible.
__global__ void __launch_bounds__(kReduceThreads)
bwd_reduce_params_kernel(const BwdArgs a, const int J) {
    stream_wait();
    __shared__ float red[kReduceThreads];
    reduce_one_param(a, J, blockIdx.x, red);
}

cudaError_t launch_reduce_params(const BwdArgs& a, int J, cudaStream_t s) {
    const int total = J * a.H + a.H + ((a.dscale_embed && a.scale_embed) ? J * a.D : 0);
    return launch_after(bwd_reduce_params_kernel, total, kReduceThreads, 0, s, a, J);
}

namespace {
template <typename T, int LPR>
cudaError_t fwd_launch(const FwdArgs& a, const Taps& t, cudaStream_t s) {
    constexpr int RPB = kFwdThreads / LPR * kFwdRows;
    dim3 grid((a.N + RPB - 1) / RPB, a.B * a.H);
    return launch_after(a.D == 4 * LPR ? fwd_generic_kernel<T, LPR, true> : fwd_generic_kernel<T, LPR, false>, grid, kFwdThreads, 0, s, a, t);
}
template <typename T>
cudaError_t fwd_launch_width(const FwdArgs& a, const Taps& t, cudaStream_t s) {
    if (a.D <= 32) return fwd_launch<T, 8>(a, t, s);
    return a.D <= 64 ? fwd_launch<T, 16>(a, t, s) : fwd_launch<T, 32>(a, t, s);
}

template <typename T, int TPR>
cudaError_t bwd_launch(BwdArgs a, const Taps& t, cudaStream_t s, int stages) {
    constexpr int RPB = kThreads / TPR;
    const bool has_se = a.scale_embed != nullptr;
    carve_bwd_scratch(a, kRowsPerBwdTile, t.J, has_se);
    size_t smem = sizeof(float) * ((size_t)RPB * t.J + RPB + (has_se ? (size_t)RPB * a.D + (size_t)t.J * a.D : 0));
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(bwd_dq_generic_kernel<T, TPR>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    cudaError_t e = cudaSuccess;
    if (stages & DSQG_BWD_STAGE_DQ) {
        dim3 grid_q(a.tiles_per_bh, a.B * a.H);
        if ((e = launch_after(bwd_dq_generic_kernel<T, TPR>, grid_q, kThreads, smem, s, a, t)) != cudaSuccess) return e;
    }
    if (stages & DSQG_BWD_STAGE_DKDV) {
        dim3 grid_k((a.N + RPB - 1) / RPB, a.B * a.H);
        if ((e = launch_after(bwd_dkdv_generic_kernel<T, TPR>, grid_k, kThreads, 0, s, a, t)) != cudaSuccess) return e;
    }
    if (stages & DSQG_BWD_STAGE_REDUCE) e = launch_reduce_params(a, t.J, s);
    return e;
}

}  // namespace

#define DSQG_DISPATCH_TPR(FN, T, ARGS, ...)                                   \
    do {                                                                      \
        const int chunks_ = (ARGS).D / 8;                                     \
        if (chunks_ <= 1) return FN<T, 1>(ARGS, __VA_ARGS__);                 \
        if (chunks_ <= 2) return FN<T, 2>(ARGS, __VA_ARGS__);                 \
        if (chunks_ <= 4) return FN<T, 4>(ARGS, __VA_ARGS__);                 \
        if (chunks_ <= 8) return FN<T, 8>(ARGS, __VA_ARGS__);                 \
        return FN<T, 16>(ARGS, __VA_ARGS__);                                  \
    } while (0)

cudaError_t launch_fwd_generic(const FwdArgs& a, const Taps& t, int dtype, cudaStream_t s) {
    return dtype == DSQG_DTYPE_BF16 ? fwd_launch_width<__nv_bfloat16>(a, t, s) : fwd_launch_width<float>(a, t, s);
}

cudaError_t launch_bwd_generic(const BwdArgs& a, const Taps& t, int dtype, cudaStream_t s, int stages) {
    if (dtype == DSQG_DTYPE_BF16) DSQG_DISPATCH_TPR(bwd_launch, __nv_bfloat16, a, t, s, stages);
    DSQG_DISPATCH_TPR(bwd_launch, float, a, t, s, stages);
}

}  // namespace dsqg
