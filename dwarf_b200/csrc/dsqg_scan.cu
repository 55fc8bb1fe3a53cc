// Causal mean along the sequence: out[b,n,:] = (x[b,0,:] + ... + x[b,n,:]) / (n + 1).
//
// This is the pooling of the DWARF condU "interference" block, which feeds the K/V injection of
// its DSQG layer: `pool = xi.cumsum(dim=1) / counts` (train/train_2048_condU.py:289-292).  The
// reference runs a cumsum in the activation dtype and a divide; here one kernel reads x once and
// writes the mean once, accumulating in fp32 whatever the storage type.
// REVERSE is its adjoint (the backward pass): out[b,n,:] = sum_{m >= n} x[b,m,:] / (m + 1).
//
// The order of the additions is part of the interface: the sequence is cut into 32 chunks of ceil(N / 32) rows, each
// chunk is summed row by row from its first, the chunk sums before a chunk (REVERSE: behind it, from the last) are added up one by
// one, and the running sum starts from there.  It depends on N alone, not on B, D, the type or the launch: the K/V deltas of a
// layer, rounded to bf16, then repeat bit for bit, and with them the gradients that nearly cancel (a bias on every key).
//
// Bound by memory; what there is to lose is loads in flight and idle SMs, since the additions of a channel are one serial chain per chunk.
// So the chains run in shared memory: all threads of a block bring the rows of its chunks there, 16 bytes each, with the
// elementwise part done on the way; one thread per chunk and channel then walks them, and all threads write the
// results.  A cluster of up to eight blocks shares 32 channels (every block stores its chunk sums in every other block's shared
// memory), so many that a block has 256 rows or four chunks.  Chunks longer than kTileRows rows are walked tile by tile and read a second time, from L2.
// No scratch memory, no atomics.  B8 N2048 D256 fp32, cold L2: 16.4 us against 53 with the same order and one thread per chunk and eight
// channels; an order that follows the launch (sums over warp and cluster first) takes 15.3.
#include "dsqg_common.cuh"

namespace dsqg {
namespace {

constexpr int kChunks = 32, kCols = 32, kScanThreads = 256, kTileRows = 128;
constexpr int kLanes = kCols / 4, kRowThreads = kScanThreads / kLanes;         // threads beside and above one another in the elementwise parts

// The gate of the interference block around the mean (train/train_2048_condU.py:289-293, fp32 mean of bf16-gated channels), so
// that its products cost no pass of their own.  Forward: inter = sigmoid(g) * mean, the sigmoid rounded to bf16 as the modules
// have it under autocast (torch.sigmoid of a bf16 projection): the K/V deltas are then theirs bit for bit.  Backward (REVERSE): the
// summands are dpool = d * sigmoid(g), and dg = d * pool * s (1 - s) is written on the way (d: gradient of inter), both with the sigmoid in fp32.
struct PoolGate {
    const __nv_bfloat16* g; const __nv_bfloat16* d; const float* pool; __nv_bfloat16* out;       // out: inter / dg
};
__device__ __forceinline__ float pool_sigmoid(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
__device__ __forceinline__ float bf16_sigmoid(float x) { return __bfloat162float(__float2bfloat16_rn(1.f / (1.f + expf(-x)))); }
// Four channels of a row.
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&x)[4]) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    x[0] = __uint_as_float(u.x << 16); x[1] = __uint_as_float(u.x & 0xffff0000u);
    x[2] = __uint_as_float(u.y << 16); x[3] = __uint_as_float(u.y & 0xffff0000u);
}
__device__ __forceinline__ void load4(const float* p, float (&x)[4]) {
    const float4 u = __ldg(reinterpret_cast<const float4*>(p));
    x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&x)[4]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]));
}
__device__ __forceinline__ void store4(float* p, const float (&x)[4]) { *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]); }

// CB: chunks of one block; 32 / CB blocks (a cluster along x) share 32 channels.  tile: rows of a chunk held at a time.
// Dynamic shared memory: [CB * tile][32] values, then [CB * tile] weights 1 / (row + 1).
template <typename T, bool REVERSE, int CB, bool GATED = false>
__global__ void __launch_bounds__(kScanThreads, 4)
causal_mean_kernel(const T* __restrict__ x, T* __restrict__ out, int N, int D, int len, int tile, const PoolGate gate) {
    stream_wait();
    constexpr int kRanks = kChunks / CB, kItems = CB * kCols, K = (kItems + kScanThreads - 1) / kScanThreads, U = GATED && REVERSE ? 2 : 4;
    extern __shared__ __align__(16) float vals[];
    __shared__ float part[kChunks][kCols];
    float* wt = vals + (size_t)CB * tile * kCols;
    if constexpr (kRanks > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");     // peers may be written to once all have started
    const int chunk0 = blockIdx.x * CB, lane4 = 4 * (threadIdx.x % kLanes), row4 = threadIdx.x / kLanes;
    const int d0 = blockIdx.y * kCols + lane4, tiles = (len + tile - 1) / tile;
    const bool active = d0 < D;
    const size_t base = (size_t)blockIdx.z * N * D + d0;
    // the rows of tile t, in turn: f(place in shared memory, row of the sequence) for U rows at a time
    auto rows_of = [&](int t, auto f) {
        const int tl = min(tile, len - t * tile), rows = active ? CB * tl : 0;
        for (int i = row4; i < rows; i += U * kRowThreads) {
            int at[U], row[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = i + u * kRowThreads, c = tiles > 1 ? k / tl : 0;         // one tile: the block's rows are consecutive
                const unsigned r = (unsigned)(chunk0 + c) * len + t * tile + (k - c * tl);
                at[u] = c * tile + (k - c * tl);
                row[u] = k < rows && r < (unsigned)N ? (int)r : -1;
            }
            f(at, row);
        }
    };
    auto load_tile = [&](int t, bool first_pass) {
        rows_of(t, [&](const int (&at)[U], const int (&row)[U]) {
            float v[U][4], g[U][4], p[U][4];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (row[u] < 0) continue;
                const size_t o = base + (size_t)row[u] * D;
                if constexpr (GATED && REVERSE) { load4(gate.d + o, v[u]); load4(gate.g + o, g[u]); load4(gate.pool + o, p[u]); }
                else load4(x + o, v[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (row[u] < 0) continue;
                if constexpr (GATED && REVERSE) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float sg = pool_sigmoid(g[u][c]);
                        p[u][c] *= v[u][c] * sg * (1.f - sg);
                        v[u][c] *= sg;
                    }
                    if (first_pass) store4(gate.out + base + (size_t)row[u] * D, p[u]);
                }
                store4(vals + at[u] * kCols + lane4, v[u]);
                if (lane4 == 0) wt[at[u]] = 1.f / (float)(row[u] + 1);
            }
        });
    };
    // the chains of this thread: channel threadIdx.x % 32 of chunks threadIdx.x / 32 + 8 k
    const int col = threadIdx.x % kCols;
    float s[K] = {};
    auto chains = [&](int t, auto f) {
        const int tl = min(tile, len - t * tile);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int c = threadIdx.x / kCols + k * (kScanThreads / kCols);
            if (c < CB) f(s[k], c * tile, max(0, min(tl, N - (chunk0 + c) * len - t * tile)));
        }
    };
    for (int t = 0; t < tiles; ++t) {
        load_tile(t, true);
        __syncthreads();
        chains(t, [&](float& sum, int at, int n) {
#pragma unroll 8
            for (int i = 0; i < n; ++i) sum = fmaf(vals[(at + i) * kCols + col], REVERSE ? wt[at + i] : 1.f, sum);
        });
        if (tiles > 1) __syncthreads();
    }
    if constexpr (kRanks > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int c = threadIdx.x / kCols + k * (kScanThreads / kCols);
        if (c >= CB) continue;
        if constexpr (kRanks > 1) {
            const uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(&part[chunk0 + c][col]));
#pragma unroll
            for (int r = 0; r < kRanks; ++r) {
                uint32_t there;
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(addr), "r"(r));
                asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(there), "f"(s[k]) : "memory");
            }
        } else {
            part[c][col] = s[k];
        }
    }
    if constexpr (kRanks > 1) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
    // what lies before (REVERSE: behind) each chunk
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int c = chunk0 + threadIdx.x / kCols + k * (kScanThreads / kCols);
        s[k] = 0.f;
        if constexpr (REVERSE) {
#pragma unroll 8
            for (int o = kChunks - 1; o > c; --o) s[k] += part[o][col];
        } else {
#pragma unroll 8
            for (int o = 0; o < min(c, kChunks); ++o) s[k] += part[o][col];
        }
    }
    for (int q = 0; q < tiles; ++q) {
        const int t = REVERSE ? tiles - 1 - q : q;
        if (tiles > 1) {
            load_tile(t, false);
            __syncthreads();
        }
        chains(t, [&](float& run, int at, int n) {
#pragma unroll 8
            for (int k = 0; k < n; ++k) {
                float& v = vals[(at + (REVERSE ? n - 1 - k : k)) * kCols + col];
                run = REVERSE ? fmaf(v, wt[at + n - 1 - k], run) : run + v;
                v = run;
            }
        });
        __syncthreads();
        rows_of(t, [&](const int (&at)[U], const int (&row)[U]) {
            float g[U][4];
            if constexpr (GATED && !REVERSE) {
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (row[u] >= 0) load4(gate.g + base + (size_t)row[u] * D, g[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (row[u] < 0) continue;
                const size_t o = base + (size_t)row[u] * D;
                const float4 v = *reinterpret_cast<const float4*>(vals + at[u] * kCols + lane4);
                const float w = REVERSE ? 1.f : wt[at[u]];
                const float y[4] = {v.x * w, v.y * w, v.z * w, v.w * w};
                store4(out + o, y);
                if constexpr (GATED && !REVERSE) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) g[u][c] = bf16_sigmoid(g[u][c]) * y[c];
                    store4(gate.out + o, g[u]);
                }
            }
        });
        if (tiles > 1) __syncthreads();
    }
}

template <typename T, bool REVERSE, bool GATED, int CB>
cudaError_t launch_scan(const T* x, T* out, int B, int N, int D, const PoolGate& gate, cudaStream_t s) {
    const int len = (N + kChunks - 1) / kChunks, tile = len < kTileRows ? len : kTileRows;
    const size_t smem = (size_t)CB * tile * (kCols + 1) * sizeof(float);
    constexpr size_t kMost = (size_t)CB * (CB == 4 ? kTileRows : 256 / CB) * (kCols + 1) * sizeof(float);
    if (smem > 48 * 1024)                                               // beyond the default limit; harmless to repeat
        if (cudaError_t e = cudaFuncSetAttribute(causal_mean_kernel<T, REVERSE, CB, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kChunks / CB, (D + kCols - 1) / kCols, B); cfg.blockDim = dim3(kScanThreads); cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kChunks / CB; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;     // as launch_after
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, causal_mean_kernel<T, REVERSE, CB, GATED>, x, out, N, D, len, tile, gate);
}

template <typename T, bool REVERSE, bool GATED = false>
cudaError_t launch_mean(const T* x, T* out, int B, int N, int D, cudaStream_t s, const PoolGate& gate = {}) {
    const int rows = (N + kChunks - 1) / kChunks;                       // of a chunk: a block gets 256 rows in all, or four chunks
    if (rows <= 8) return launch_scan<T, REVERSE, GATED, 32>(x, out, B, N, D, gate, s);
    if (rows <= 16) return launch_scan<T, REVERSE, GATED, 16>(x, out, B, N, D, gate, s);
    if (rows <= 32) return launch_scan<T, REVERSE, GATED, 8>(x, out, B, N, D, gate, s);
    return launch_scan<T, REVERSE, GATED, 4>(x, out, B, N, D, gate, s);
}

}  // namespace

cudaError_t launch_gated_mean(const float* x, const void* g, float* pool, void* inter, int B, int N, int D, cudaStream_t s) {
    return launch_mean<float, false, true>(x, pool, B, N, D, s, {static_cast<const __nv_bfloat16*>(g), nullptr, nullptr, static_cast<__nv_bfloat16*>(inter)});
}
cudaError_t launch_gated_mean_bwd(const void* dinter, const void* g, const float* pool, void* dg, float* dx, int B, int N, int D, cudaStream_t s) {
    return launch_mean<float, true, true>(nullptr, dx, B, N, D, s, {static_cast<const __nv_bfloat16*>(g), static_cast<const __nv_bfloat16*>(dinter), pool,
                                                                    static_cast<__nv_bfloat16*>(dg)});
}

cudaError_t launch_causal_mean(const void* x, void* out, int B, int N, int D, int dtype, bool reverse, cudaStream_t s) {
    if (dtype == DSQG_DTYPE_BF16) {
        auto xi = static_cast<const __nv_bfloat16*>(x); auto oi = static_cast<__nv_bfloat16*>(out);
        return reverse ? launch_mean<__nv_bfloat16, true>(xi, oi, B, N, D, s) : launch_mean<__nv_bfloat16, false>(xi, oi, B, N, D, s);
    }
    auto xi = static_cast<const float*>(x); auto oi = static_cast<float*>(out);
    return reverse ? launch_mean<float, true>(xi, oi, B, N, D, s) : launch_mean<float, false>(xi, oi, B, N, D, s);
}

}  // namespace dsqg
