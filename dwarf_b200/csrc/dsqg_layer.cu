// What an attention layer does between its GEMMs and the DSQG operator, one pass over memory each.
//
// A condU layer with the interference block (DWARF train/train_2048_condU.py:171-191, 277-295) under bf16 autocast is
// about ninety PyTorch launches per step: weight and activation casts, layer norm and its two backward kernels,
// sigmoids, products, K/V additions, bias sums.  These kernels are the parts that are left when every tensor is read and
// written once.  All of them are bound by memory (or by the launch, at small sizes); fp32 arithmetic throughout.
#include "dsqg_common.cuh"

namespace dsqg {
namespace {

constexpr int kT = 256;

// ---- fp32 -> bf16 for up to kCastMax tensors in one launch
struct CastArgs { const float* src[DSQG_CAST_MAX]; __nv_bfloat16* dst[DSQG_CAST_MAX]; long long end[DSQG_CAST_MAX]; int count; };   // end: running sum of the lengths

__global__ void __launch_bounds__(kT) cast_kernel(const CastArgs a) {
    stream_wait();
    const long long total = a.end[a.count - 1];
    for (long long i = ((long long)blockIdx.x * kT + threadIdx.x) * 8; i < total; i += (long long)gridDim.x * kT * 8) {
        int k = 0;
        while (i >= a.end[k]) ++k;
        const long long o = i - (k ? a.end[k - 1] : 0);
        float x[8];
        load8(a.src[k] + o, x);
        store8(a.dst[k] + o, x);
    }
}

// ---- layer norm forward: one warp per row.  y in fp32 (for the running mean) and bf16 (for the GEMM).  For callers of the C interface (29 us at
// 65,536 x 256); the autograd node of the interference block takes PyTorch's kernel (112 us, and a cast), whose last bits its deltas follow.
__global__ void __launch_bounds__(kT)
layer_norm_fwd_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta, float eps,
                      float* __restrict__ y, __nv_bfloat16* __restrict__ yb, float2* __restrict__ stat, long long rows, int D) {
    stream_wait();
    const long long row = (long long)blockIdx.x * (kT / 32) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    const float* xr = x + row * D;
    float s = 0.f;
    for (int c = 4 * lane; c < D; c += 128) {
        const float4 v = *reinterpret_cast<const float4*>(xr + c);
        s += (v.x + v.y) + (v.z + v.w);
    }
    const float mean = group_sum<32>(s) / D;
    float q = 0.f;
    for (int c = 4 * lane; c < D; c += 128) {                 // the row is in L1 by now
        const float4 v = *reinterpret_cast<const float4*>(xr + c);
        const float a = v.x - mean, b = v.y - mean, e = v.z - mean, f = v.w - mean;
        q += (a * a + b * b) + (e * e + f * f);
    }
    const float rstd = rsqrtf(group_sum<32>(q) / D + eps);
    if (lane == 0) stat[row] = make_float2(mean, rstd);
    for (int c = 4 * lane; c < D; c += 128) {
        const float4 v = *reinterpret_cast<const float4*>(xr + c), g = *reinterpret_cast<const float4*>(gamma + c);
        const float4 b = *reinterpret_cast<const float4*>(beta + c);
        const float4 o = make_float4(fmaf((v.x - mean) * rstd, g.x, b.x), fmaf((v.y - mean) * rstd, g.y, b.y),
                                     fmaf((v.z - mean) * rstd, g.z, b.z), fmaf((v.w - mean) * rstd, g.w, b.w));
        *reinterpret_cast<float4*>(y + row * D + c) = o;
        *reinterpret_cast<uint2*>(yb + row * D + c) = make_uint2(pack_bf16x2(o.x, o.y), pack_bf16x2(o.z, o.w));
    }
}

// ---- layer norm backward with dy = dya (fp32) + dyb (bf16): dx, and per-block partial sums of dgamma / dbeta.
// mean, rstd: `step` elements from row to row.  One warp per row, each warp walks rows a grid apart; a lane keeps the sums of its columns (at most 32: D <= 1024).
// Bound by memory, and there by loads in flight: up to 256 columns a warp brings R = 2 rows at once (94 registers, two blocks an SM as before).
// With the reduction of the partials, L2 cold, D 256: 65,536 rows 61.7 -> 47.0 us (HBM's floor 36), 16,384 rows 22.2 -> 20.9; three rows 48.3 and
// 23.2, three blocks an SM instead 60.6 and 26.4.  The order of the sums, and with it every bit, is that of one row at a time.
template <int C4>
__global__ void __launch_bounds__(kT)
layer_norm_bwd_kernel(const float* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ rstd, int step, const float* __restrict__ gamma,
                      const float* __restrict__ dya, const __nv_bfloat16* __restrict__ dyb, float* __restrict__ dx,
                      float* __restrict__ part, long long rows, int D) {
    stream_wait();
    extern __shared__ float sums[];                            // [2][D]
    constexpr int R = C4 <= 2 ? 2 : 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4 dg[C4], db[C4];
#pragma unroll
    for (int i = 0; i < C4; ++i) dg[i] = db[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const long long stride = (long long)gridDim.x * (kT / 32);
    for (long long row0 = (long long)blockIdx.x * (kT / 32) + warp; row0 < rows; row0 += R * stride) {
        float4 v[R][C4], d[R][C4];
        uint2 u[R][C4];
        float2 st[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long long row = row0 + r * stride;
            if (row >= rows) break;
            st[r] = make_float2(__ldg(mean + row * step), __ldg(rstd + row * step));
#pragma unroll
            for (int i = 0; i < C4; ++i) {
                const int c = 4 * lane + 128 * i;
                if (c >= D) break;
                v[r][i] = __ldg(reinterpret_cast<const float4*>(x + row * D + c));
                d[r][i] = __ldg(reinterpret_cast<const float4*>(dya + row * D + c));
                u[r][i] = __ldg(reinterpret_cast<const uint2*>(dyb + row * D + c));
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long long row = row0 + r * stride;
            if (row >= rows) break;
            const float mu = st[r].x, rs = st[r].y;
            float s1 = 0.f, s2 = 0.f;
            // v and d become x^ and dy gamma
#pragma unroll
            for (int i = 0; i < C4; ++i) {
                const int c = 4 * lane + 128 * i;
                if (c >= D) break;
                float4 &xh = v[r][i], &w = d[r][i];
                w.x += __uint_as_float(u[r][i].x << 16); w.y += __uint_as_float(u[r][i].x & 0xffff0000u);
                w.z += __uint_as_float(u[r][i].y << 16); w.w += __uint_as_float(u[r][i].y & 0xffff0000u);
                const float4 g = __ldg(reinterpret_cast<const float4*>(gamma + c));
                xh = make_float4((xh.x - mu) * rs, (xh.y - mu) * rs, (xh.z - mu) * rs, (xh.w - mu) * rs);
                dg[i].x = fmaf(w.x, xh.x, dg[i].x); dg[i].y = fmaf(w.y, xh.y, dg[i].y);
                dg[i].z = fmaf(w.z, xh.z, dg[i].z); dg[i].w = fmaf(w.w, xh.w, dg[i].w);
                db[i].x += w.x; db[i].y += w.y; db[i].z += w.z; db[i].w += w.w;
                w = make_float4(w.x * g.x, w.y * g.y, w.z * g.z, w.w * g.w);
                s1 += (w.x + w.y) + (w.z + w.w);
                s2 += (w.x * xh.x + w.y * xh.y) + (w.z * xh.z + w.w * xh.w);
            }
            s1 = group_sum<32>(s1) / D; s2 = group_sum<32>(s2) / D;
#pragma unroll
            for (int i = 0; i < C4; ++i) {
                const int c = 4 * lane + 128 * i;
                if (c >= D) break;
                const float4 &xh = v[r][i], &w = d[r][i];
                *reinterpret_cast<float4*>(dx + row * D + c) =
                    make_float4(rs * (w.x - s1 - xh.x * s2), rs * (w.y - s1 - xh.y * s2), rs * (w.z - s1 - xh.z * s2), rs * (w.w - s1 - xh.w * s2));
            }
        }
    }
    for (int w = 0; w < kT / 32; ++w) {                        // warps in turn: fixed order of additions
        if (warp == w) {
#pragma unroll
            for (int i = 0; i < C4; ++i) {
                const int c = 4 * lane + 128 * i;
                if (c >= D) break;
                const float a[4] = {dg[i].x, dg[i].y, dg[i].z, dg[i].w}, b[4] = {db[i].x, db[i].y, db[i].z, db[i].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    sums[c + e] = w ? sums[c + e] + a[e] : a[e];
                    sums[D + c + e] = w ? sums[D + c + e] + b[e] : b[e];
                }
            }
        }
        __syncthreads();
    }
    for (int c = threadIdx.x; c < 2 * D; c += kT) part[(size_t)blockIdx.x * 2 * D + c] = sums[c];
}

// out[c] = sum_b part[b][c], one warp per 32 columns, rows of the table split over the warps of a block
__global__ void __launch_bounds__(kT) sum_rows_kernel(const float* __restrict__ part, float* __restrict__ out, int n, int C) {
    stream_wait();
    __shared__ float red[kT / 32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (c < C) {
#pragma unroll 8
        for (int b = warp; b < n; b += kT / 32) s += part[(size_t)b * C + c];
    }
    red[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && c < C) {
        s = 0.f;
#pragma unroll
        for (int w = 0; w < kT / 32; ++w) s += red[w][lane];
        out[c] = s;
    }
}

// ---- k += k_delta, v += v_delta on columns D .. 3 D of qkv; rows lq / ld elements apart
__global__ void __launch_bounds__(kT) inject_kernel(__nv_bfloat16* __restrict__ qkv, long long lq, const __nv_bfloat16* __restrict__ kd,
                                                    const __nv_bfloat16* __restrict__ vd, long long ld, long long rows, int D) {
    stream_wait();
    const long long i = (long long)blockIdx.x * kT + threadIdx.x;
    const int per = D / 8;                                     // 16-byte pieces of a delta row
    if (i >= rows * 2 * per) return;
    const long long row = i / (2 * per);
    const int c = (int)(i - row * 2 * per);
    __nv_bfloat16* dst = qkv + row * lq + D + 8 * c;
    float x[8], y[8];
    load8(dst, x); load8((c < per ? kd + 8 * c : vd + 8 * (c - per)) + row * ld, y);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] += y[e];
    store8(dst, x);
}

// ---- column sums of up to DSQG_SUM_MAX bf16 matrices [rows][cols] in one launch (bias gradients).  A cluster of eight blocks
// takes 64 columns (a 128-byte line of every row); each block adds an eighth of the rows, block 0 adds the eight results.
struct SumArgs { const __nv_bfloat16* src[DSQG_SUM_MAX]; float* dst[DSQG_SUM_MAX]; long long ld[DSQG_SUM_MAX]; int slice_end[DSQG_SUM_MAX], cols[DSQG_SUM_MAX]; int count; long long rows; };
constexpr int kSumThreads = 512, kSumCols = 64, kSumRows = kSumThreads / (kSumCols / 8);

__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(kSumThreads) column_sum_kernel(const SumArgs a) {
    stream_wait();
    __shared__ float red[kSumRows][kSumCols + 1];
    __shared__ float total[8][kSumCols];
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");      // block 0 may be written to once it has started
    int k = 0;
    while ((int)blockIdx.y >= a.slice_end[k]) ++k;
    const int c0 = ((int)blockIdx.y - (k ? a.slice_end[k - 1] : 0)) * kSumCols, c = threadIdx.x % (kSumCols / 8) * 8, r = threadIdx.x / (kSumCols / 8);
    const long long per = (a.rows + 7) / 8, first = blockIdx.x * per, last = min(a.rows, first + per);
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (c0 + c < a.cols[k]) {
        const __nv_bfloat16* p = a.src[k] + c0 + c;
#pragma unroll 8
        for (long long i = first + r; i < last; i += kSumRows) {
            float x[8];
            load8(p + i * a.ld[k], x);
#pragma unroll
            for (int e = 0; e < 8; ++e) s[e] += x[e];
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) red[r][c + e] = s[e];
    __syncthreads();
    const int col = threadIdx.x % kSumCols, part = threadIdx.x / kSumCols;          // eight parts of eight rows
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += red[part * 8 + i][col];
    __syncthreads();
    red[part][col] = t;
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (part == 0) {
        t = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += red[i][col];
        uint32_t there;
        const uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(&total[blockIdx.x][col]));
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(addr), "r"(0));
        asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(there), "f"(t) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (blockIdx.x == 0 && part == 0 && c0 + col < a.cols[k]) {
        t = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += total[i][col];
        a.dst[k][c0 + col] = t;
    }
}

inline unsigned blocks_for(long long n) { return (unsigned)((n + kT - 1) / kT); }
constexpr int kNormBlocks = 148 * 2;
inline unsigned norm_blocks(long long rows) { const long long b = (rows + kT / 32 - 1) / (kT / 32); return (unsigned)(b < kNormBlocks ? b : kNormBlocks); }
inline bool bad(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) != 0; }
inline int status(cudaError_t e) { return e == cudaSuccess ? DSQG_OK : DSQG_ERR_CUDA; }
inline bool bad_rows(long long rows, int D) { return rows < 1 || D < 8 || D % 8 || D > 1024 || rows * D > 0x7fffffffffLL; }

}  // namespace
}  // namespace dsqg

using namespace dsqg;

extern "C" {

int dsqg_cast_bf16(const float* const* src, void* const* dst, const long long* n, int count, void* stream) {
    if (!src || !dst || !n) return DSQG_ERR_NULL_POINTER;
    if (count < 1 || count > DSQG_CAST_MAX) return DSQG_ERR_BAD_SHAPE;
    CastArgs a;
    a.count = count;
    long long total = 0;
    for (int k = 0; k < count; ++k) {
        if (!src[k] || !dst[k]) return DSQG_ERR_NULL_POINTER;
        if (n[k] < 8 || n[k] % 8) return DSQG_ERR_BAD_SHAPE;
        if (bad(src[k]) || bad(dst[k])) return DSQG_ERR_MISALIGNED;
        a.src[k] = src[k]; a.dst[k] = static_cast<__nv_bfloat16*>(dst[k]); a.end[k] = total += n[k];
    }
    const unsigned blocks = blocks_for(total / 8);
    return status(launch_after(cast_kernel, blocks < 148 * 16 ? blocks : 148 * 16, kT, 0, static_cast<cudaStream_t>(stream), a));
}

int dsqg_layer_norm_fwd(const float* x, const float* gamma, const float* beta, float eps, float* y, void* y_bf16, float* stat,
                        long long rows, int D, void* stream) {
    if (!x || !gamma || !beta || !y || !y_bf16 || !stat) return DSQG_ERR_NULL_POINTER;
    if (bad_rows(rows, D)) return DSQG_ERR_BAD_SHAPE;
    if (bad(x) || bad(gamma) || bad(beta) || bad(y) || bad(y_bf16) || bad(stat)) return DSQG_ERR_MISALIGNED;
    return status(launch_after(layer_norm_fwd_kernel, (unsigned)((rows + kT / 32 - 1) / (kT / 32)), kT, 0, static_cast<cudaStream_t>(stream),
        x, gamma, beta, eps, y, static_cast<__nv_bfloat16*>(y_bf16), reinterpret_cast<float2*>(stat), rows, D));
}

size_t dsqg_layer_norm_bwd_scratch_bytes(long long rows, int D) {
    return bad_rows(rows, D) ? 0 : (size_t)norm_blocks(rows) * 2 * D * 4;
}

static int norm_bwd(const float* x, const float* mean, const float* rstd, int step, const float* gamma, const float* dy, const void* dy_bf16, float* dx,
                    float* dgamma_dbeta, void* scratch, size_t scratch_bytes, long long rows, int D, void* stream) {
    if (!x || !mean || !rstd || !gamma || !dy || !dy_bf16 || !dx || !dgamma_dbeta || !scratch) return DSQG_ERR_NULL_POINTER;
    if (bad_rows(rows, D)) return DSQG_ERR_BAD_SHAPE;
    if (bad(x) || bad(gamma) || bad(dy) || bad(dy_bf16) || bad(dx) || bad(dgamma_dbeta) || bad(scratch)) return DSQG_ERR_MISALIGNED;
    if (scratch_bytes < dsqg_layer_norm_bwd_scratch_bytes(rows, D)) return DSQG_ERR_SCRATCH_TOO_SMALL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const unsigned blocks = norm_blocks(rows);
    const size_t smem = (size_t)2 * D * 4;
    float* part = static_cast<float*>(scratch);
    const __nv_bfloat16* db = static_cast<const __nv_bfloat16*>(dy_bf16);
    auto kern = D <= 256 ? layer_norm_bwd_kernel<2> : (D <= 512 ? layer_norm_bwd_kernel<4> : layer_norm_bwd_kernel<8>);
    if (int rc = status(launch_after(kern, blocks, kT, smem, s, x, mean, rstd, step, gamma, dy, db, dx, part, rows, D))) return rc;
    return status(launch_after(sum_rows_kernel, (2 * D + 31) / 32, kT, 0, s, part, dgamma_dbeta, (int)blocks, 2 * D));
}

int dsqg_layer_norm_bwd(const float* x, const float* stat, const float* gamma, const float* dy, const void* dy_bf16, float* dx,
                        float* dgamma_dbeta, void* scratch, size_t scratch_bytes, long long rows, int D, void* stream) {
    if (!stat) return DSQG_ERR_NULL_POINTER;
    if (bad(stat)) return DSQG_ERR_MISALIGNED;
    return norm_bwd(x, stat, stat + 1, 2, gamma, dy, dy_bf16, dx, dgamma_dbeta, scratch, scratch_bytes, rows, D, stream);
}

int dsqg_layer_norm_bwd_split(const float* x, const float* mean, const float* rstd, const float* gamma, const float* dy, const void* dy_bf16, float* dx,
                              float* dgamma_dbeta, void* scratch, size_t scratch_bytes, long long rows, int D, void* stream) {
    return norm_bwd(x, mean, rstd, 1, gamma, dy, dy_bf16, dx, dgamma_dbeta, scratch, scratch_bytes, rows, D, stream);
}

int dsqg_gated_mean(const float* x, const void* g, float* pool, void* inter, int B, int N, int D, void* stream) {
    if (!x || !g || !pool || !inter) return DSQG_ERR_NULL_POINTER;
    if (B < 1 || B > 65535 || N < 1 || D < 8 || D % 8) return DSQG_ERR_BAD_SHAPE;
    if (bad(x) || bad(g) || bad(pool) || bad(inter)) return DSQG_ERR_MISALIGNED;
    return launch_gated_mean(x, g, pool, inter, B, N, D, static_cast<cudaStream_t>(stream)) == cudaSuccess ? DSQG_OK : DSQG_ERR_CUDA;
}

int dsqg_gated_mean_bwd(const void* dinter, const void* g, const float* pool, void* dg, float* dx, int B, int N, int D, void* stream) {
    if (!dinter || !g || !pool || !dg || !dx) return DSQG_ERR_NULL_POINTER;
    if (B < 1 || B > 65535 || N < 1 || D < 8 || D % 8) return DSQG_ERR_BAD_SHAPE;
    if (bad(dinter) || bad(g) || bad(pool) || bad(dg) || bad(dx)) return DSQG_ERR_MISALIGNED;
    return launch_gated_mean_bwd(dinter, g, pool, dg, dx, B, N, D, static_cast<cudaStream_t>(stream)) == cudaSuccess ? DSQG_OK : DSQG_ERR_CUDA;
}

int dsqg_inject_kv(void* qkv, long long qkv_stride, const void* k_delta, const void* v_delta, long long delta_stride, long long rows, int D, void* stream) {
    if (!qkv || !k_delta || !v_delta) return DSQG_ERR_NULL_POINTER;
    if (rows < 1 || D < 8 || D % 8) return DSQG_ERR_BAD_SHAPE;
    if (bad(qkv) || bad(k_delta) || bad(v_delta) || delta_stride < D || delta_stride % 8 || qkv_stride < 3 * D || qkv_stride % 8) return DSQG_ERR_MISALIGNED;
    return status(launch_after(inject_kernel, blocks_for(rows * (D / 4)), kT, 0, static_cast<cudaStream_t>(stream),
        static_cast<__nv_bfloat16*>(qkv), qkv_stride, static_cast<const __nv_bfloat16*>(k_delta), static_cast<const __nv_bfloat16*>(v_delta), delta_stride, rows, D));
}

int dsqg_column_sums(const void* const* src, const long long* row_stride, const int* cols, float* const* dst, int count, long long rows, void* stream) {
    if (!src || !row_stride || !cols || !dst) return DSQG_ERR_NULL_POINTER;
    if (count < 1 || count > DSQG_SUM_MAX || rows < 1) return DSQG_ERR_BAD_SHAPE;
    SumArgs a;
    a.count = count; a.rows = rows;
    int slices = 0;
    for (int k = 0; k < count; ++k) {
        if (!src[k] || !dst[k]) return DSQG_ERR_NULL_POINTER;
        if (cols[k] < 8 || cols[k] % 8) return DSQG_ERR_BAD_SHAPE;
        if (bad(src[k]) || row_stride[k] < cols[k] || row_stride[k] % 8) return DSQG_ERR_MISALIGNED;
        a.src[k] = static_cast<const __nv_bfloat16*>(src[k]); a.dst[k] = dst[k]; a.ld[k] = row_stride[k]; a.cols[k] = cols[k];
        a.slice_end[k] = slices += (cols[k] + kSumCols - 1) / kSumCols;
    }
    if (slices > 65535) return DSQG_ERR_BAD_SHAPE;
    return status(launch_after(column_sum_kernel, dim3(8, slices), kSumThreads, 0, static_cast<cudaStream_t>(stream), a));
}

}  // extern "C"
