// Weight and bias gradients of a layer's projections on the 5th-generation tensor cores: dW = dY^T . X in fp32 and the column
// sums of dY, up to two products of one contraction length in one launch (bf16 operands, sm_100a).
//
// Reference math: nn.Linear's backward for the projections of DWARF train/train_2048_condU.py:171-191, :277-295.
//
// The outputs are small (256 x 256 to 1024 x 256) and the contraction is long (batch x sequence), so the contraction is what
// is split: a cluster of up to eight blocks shares one 128 x 128 or 128 x 256 tile of dW, each block takes a range of rows of dY and X and
// the fp32 partial tiles are added over distributed shared memory, block 0's first: fixed order, no scratch, no second pass.
// Both operands lie with the contraction as their slow dimension; they are staged as 64-row boxes of 64 columns (128 bytes, one
// swizzle atom) and enter tcgen05.mma as MN-major tiles, so nothing is transposed.  Warps 0-3 add dY's columns from the staged
// tile while the tensor cores work on it, which costs no second pass over dY.
//   warp 4 (one lane): copies (cp.async.bulk.tensor, four or six stages of 64 rows)    warp 5 (one lane): tcgen05.mma, M 128, N 128 or 256
//   warps 0-3: column sums, then accumulators -> shared memory (over the stages)    all: a share of the cluster's sum -> dW
// Every wait is bounded (stg::mbar_wait).  A block that gives up sets the device error word and the one in host memory, which the next call
// looks at, and its cluster writes NaN to its part of dW and of the sums; copies and products in flight are waited for all the same.
//
// Bound by what an SM can fetch (90 GB/s a block measured, from L2 or HBM; all 148 together would outrun HBM): [1024, 256] + [256, 256]
// gradients with their sums, against two library GEMMs and a pass for the sums: 4,096 rows 11.0 us : 18.5, 16,384 23.1 : 49.5, 65,536
// 70 : 107 (HBM's floor there 36).  A tile of 128 x 256 with eight blocks a cluster took 25 and 72 us for the first two products, but
// 24 and 70 instead of 18.7 and 54 for [512, 256] + [256, 256], whose six tiles leave most of the chip idle: hence two widths.  The sums cost 6 of
// the 70 us (shared-memory reads beside the tensor cores'); added by one tile in two instead of half by each they cost 10.
#include <cuda.h>
#include <cuda_bf16.h>

#include <mutex>

#include "dsqg_common.cuh"
#include "dsqg_stage.cuh"
#include "dsqg_tcgen05.cuh"

namespace dsqg {
namespace wgrad {

using namespace stg;
using namespace tc5;

constexpr int kTM = 128;                       // columns of dY of a tile
constexpr int kBox = 64;                       // rows and columns of a staged box
constexpr int kBoxBytes = kBox * 128;
constexpr int kThreads = 192, kCopyWarp = 4, kMmaWarp = 5;
constexpr int kMostSplit = 8;
constexpr long long kLimit = 4000000000LL;      // cycles before a wait gives up: two seconds, far above any time slice of a shared GPU
// TN: columns of X of a tile
template <int TN>
struct Layout {
    static constexpr int a_bytes = kTM / kBox * kBoxBytes, stage_bytes = a_bytes + TN / kBox * kBoxBytes;      // 48 / 32 KB
    static constexpr int stages = 192 * 1024 / stage_bytes;
    static constexpr int pitch = TN + 4;                           // floats per row of the partial tile (16-byte stores of neighbouring rows: other banks)
    static constexpr int sum0 = stages * stage_bytes;              // column sums of 8 row classes x kTM columns or 16 x 64, then their total [kTM]
    static constexpr int bars0 = sum0 + (8 + 1) * kTM * 4;
    static constexpr int full = 0, empty = stages, done = 2 * stages, bars = done + 1;
    static constexpr int total = bars0 + 256 + 1024;               // 1,024: alignment of the swizzle atoms
    static_assert(kTM * pitch * 4 <= sum0, "the partial tile lies over the stages");
    // fp32 accumulator, bf16 A and B, both MN-major
    static constexpr uint32_t instr = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(kTM >> 4) << 24);
};

static_assert(DSQG_WGRAD_MAX == 2, "two jobs, four tensor maps");
struct Job { int cols, tiles_end; float* dw; float* sum; bool a_hf, b_hf; };
struct Args { Job job[DSQG_WGRAD_MAX]; int rows, D, split; int* report; long long limit; };       // limit: cycles before a wait gives up

__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t there;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(addr), "r"(rank));
    return there;
}
__device__ __forceinline__ float4 cluster_load4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float cluster_load(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ int cluster_load_int(uint32_t addr) {
    int v;
    asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 128-byte-swizzled tile of MN-major boxes: 64-column boxes kBoxBytes apart, groups of eight contraction rows 1,024 bytes apart.
__device__ __forceinline__ uint64_t mn_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(kBoxBytes >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// STALL: the last block of every cluster never asks for the second half of its rows, so that waits run out (dsqg_test_weight_grads_timeout).
template <int TN, bool STALL = false>
__global__ void __launch_bounds__(kThreads, 1)
weight_grad_kernel(const Args a, const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_b0,
                   const __grid_constant__ CUtensorMap map_a1, const __grid_constant__ CUtensorMap map_b1) {
    using L = Layout<TN>;
    constexpr int kStages = L::stages, kStageBytes = L::stage_bytes, kABytes = L::a_bytes, kSum0 = L::sum0, kBars0 = L::bars0, kNumBars = L::bars,
                  kFull = L::full, kEmpty = L::empty, kDone = L::done, kPitch = L::pitch;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sb = smem_u32(smem), bars = sb + kBars0;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kBars0 + 8 * kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kBars0 + 8 * kNumBars + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x % a.split, tile = blockIdx.x / a.split;
    const int j = tile >= a.job[0].tiles_end ? 1 : 0;
    const Job job = j ? a.job[1] : a.job[0];
    const int across = (a.D + TN - 1) / TN, in_job = tile - (j ? a.job[0].tiles_end : 0);
    const int c0 = in_job / across * kTM, k0 = in_job % across * TN;
    // dY's columns are added by the tiles of the first columns of X: all 128 by one, or 64 each by two
    const bool halves = across > 1, sums = job.sum && k0 < (halves ? 2 * TN : TN);
    const int sum_cols = halves ? 64 : kTM, sum_c = halves ? k0 / TN * 64 : 0;
    const int blocks = (a.rows + kBox - 1) / kBox;
    const int first = (int)((long long)blocks * rank / a.split), count = (int)((long long)blocks * (rank + 1) / a.split) - first;

    // tensor memory is asked for when nothing of the kernel ahead holds or still wants any, and before the next kernel may: two kernels
    // that wait for each other's columns would wait for good
    wait_ahead();
    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < kStages; ++i) { mbar_init(bars + 8 * (kFull + i), 1); mbar_init(bars + 8 * (kEmpty + i), sums ? 5 : 1); }
        mbar_init(bars + 8 * kDone, 1);
        fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(tmem_slot), TN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    let_next_in();

    if (warp == kCopyWarp) {
        if (lane == 0) {
            const Tma ta = {j ? &map_a1 : &map_a0, job.a_hf}, tb = {j ? &map_b1 : &map_b0, job.b_hf};
            const int copies = STALL && rank == a.split - 1 ? count / 2 : count;
            int i = 0;
            for (; i < copies; ++i) {
                const int st = i % kStages;
                if (i >= kStages && !mbar_wait(bars + 8 * (kEmpty + st), (i / kStages - 1) & 1, abort_flag, 0x501, a.limit, a.report)) break;
                const uint32_t bar = bars + 8 * (kFull + st), dst = sb + st * kStageBytes;
                const int row = (first + i) * kBox;
                mbar_arrive_expect_tx(bar, kStageBytes);               // boxes outside a matrix arrive as zeros
#pragma unroll
                for (int b = 0; b < kTM / kBox; ++b) ta.load(dst + b * kBoxBytes, bar, row, c0 / kBox + b, 0);
#pragma unroll
                for (int b = 0; b < TN / kBox; ++b) tb.load(dst + kABytes + b * kBoxBytes, bar, row, k0 / kBox + b, 0);
            }
            // no copy may be in flight when the shared memory is released, whoever gave up and when: a flag of its own
            volatile int keep_waiting = 0;
            for (int k = i > kStages ? i - kStages : 0; k < i; ++k) mbar_wait(bars + 8 * (kFull + k % kStages), (k / kStages) & 1, &keep_waiting, 0x504, kLimit, a.report);
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        if (lane == 0) {
            const uint64_t desc0 = mn_desc(sb);
            for (int i = 0; i < count; ++i) {
                const int st = i % kStages;
                if (!mbar_wait(bars + 8 * (kFull + st), (i / kStages) & 1, abort_flag, 0x502, a.limit, a.report)) break;
                tc_fence_after();
                const uint64_t da = desc0 + (uint32_t)(st * kStageBytes >> 4), db = da + (uint32_t)(kABytes >> 4);
#pragma unroll
                for (int kk = 0; kk < kBox / 16; ++kk)                 // 16 contraction rows = two groups of eight
                    umma_bf16(tmem, da + kk * (2048 >> 4), db + kk * (2048 >> 4), L::instr, i > 0 || kk > 0);
                umma_commit(bars + 8 * (kEmpty + st));
            }
            umma_commit(bars + 8 * kDone);
            volatile int keep_waiting = 0;                             // as above: no product when the tensor memory is released
            mbar_wait(bars + 8 * kDone, 0, &keep_waiting, 0x506, kLimit, a.report);
        }
        __syncwarp();
    } else {
        float* csum = reinterpret_cast<float*>(smem + kSum0);
        if (sums) {
            // thread: eight columns (one 16-byte chunk) of every 8th or 16th row of a stage; the chunk index is XORed with row & 7
            const int chunk = tid & 7, half = halves ? sum_c / 64 : tid >> 3 & 1, r = tid >> (halves ? 3 : 4), apart = halves ? 16 : 8;
            const unsigned char* src = smem + half * kBoxBytes + r * 128 + ((chunk ^ (r & 7)) << 4);
            float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int i = 0; i < count; ++i) {
                const int st = i % kStages;
                if (!__all_sync(0xffffffffu, mbar_wait(bars + 8 * (kFull + st), (i / kStages) & 1, abort_flag, 0x503, a.limit, a.report))) break;
                uint4 u[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    u[k] = k < 4 || !halves ? *reinterpret_cast<const uint4*>(src + st * kStageBytes + k * apart * 128) : make_uint4(0u, 0u, 0u, 0u);
                __syncwarp();
                if (lane == 0) mbar_arrive(bars + 8 * (kEmpty + st));
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (k >= 4 && halves) break;
                    const uint32_t w[4] = {u[k].x, u[k].y, u[k].z, u[k].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) { s[2 * e] += __uint_as_float(w[e] << 16); s[2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u); }
                }
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) csum[r * sum_cols + (halves ? 0 : half * 64) + chunk * 8 + e] = s[e];
            asm volatile("bar.sync 1, 128;" ::: "memory");
            float t = 0.f;
            if (tid < sum_cols)
                for (int k = 0; k < apart; ++k) t += csum[k * sum_cols + tid];
            csum[8 * kTM + tid] = t;
        }
        // accumulator row = tensor-memory lane = tid; the stages are free once every product has completed
        const bool ok = __all_sync(0xffffffffu, mbar_wait(bars + 8 * kDone, 0, abort_flag, 0x505, a.limit, a.report) && !*abort_flag);
        tc_fence_after();
        float* part = reinterpret_cast<float*>(smem) + tid * kPitch;
        const uint32_t acc = tmem + ((uint32_t)(32 * warp) << 16);
        if (sums) asm volatile("bar.sync 1, 128;" ::: "memory");
        if (ok) {
#pragma unroll 1
            for (int c = 0; c < TN; c += 32) {
                float v[32];
                tmem_ld32(v, acc + c);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 8; ++e) *reinterpret_cast<float4*>(part + c + 4 * e) = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
            }
        }
        tc_fence_before();
    }
    cluster_sync();

    // rows [128 rank / split, 128 (rank + 1) / split) of the tile: the cluster's partial tiles, in block order
    {
        const int r0 = kTM * rank / a.split, r1 = kTM * (rank + 1) / a.split;
        const int rows = min(r1, job.cols - c0) - r0, wide = min(TN, a.D - k0) / 4;
        uint32_t base[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) base[b] = cluster_addr(sb, b < a.split ? b : 0);
        const int gave_up = lane < a.split ? cluster_load_int(cluster_addr(sb + kBars0 + 8 * kNumBars + 8, lane)) : 0;      // the blocks' abort_flag
        for (int e = tid; e < rows * wide; e += kThreads) {
            const int r = r0 + e / wide, c = e % wide * 4;
            const uint32_t off = (uint32_t)(r * kPitch + c) * 4;
            float4 v[8], t;
#pragma unroll
            for (int b = 0; b < 8; ++b) if (b < a.split) v[b] = cluster_load4(base[b] + off);
            t = v[0];
#pragma unroll
            for (int b = 1; b < 8; ++b) if (b < a.split) { t.x += v[b].x; t.y += v[b].y; t.z += v[b].z; t.w += v[b].w; }
            *reinterpret_cast<float4*>(job.dw + (size_t)(c0 + r) * a.D + k0 + c) = t;
        }
        if (sums && rank == 0 && tid < min(sum_cols, job.cols - c0 - sum_c)) {
            float t = 0.f;
            for (int b = 0; b < a.split; ++b) t += cluster_load(cluster_addr(sb + kSum0 + (8 * kTM + tid) * 4, b));
            job.sum[c0 + sum_c + tid] = t;
        }
        if (__any_sync(0xffffffffu, gave_up)) {                        // each thread over what it wrote itself
            const float nan = __int_as_float(0x7fffffff);
            for (int e = tid; e < rows * wide; e += kThreads)
                *reinterpret_cast<float4*>(job.dw + (size_t)(c0 + r0 + e / wide) * a.D + k0 + e % wide * 4) = make_float4(nan, nan, nan, nan);
            if (sums && rank == 0 && tid < min(sum_cols, job.cols - c0 - sum_c)) job.sum[c0 + sum_c + tid] = nan;
        }
    }
    cluster_sync();                                                    // nobody's shared memory goes while others read it
    tc_fence_after();
    if (warp == kMmaWarp) tmem_dealloc(tmem, TN);
}

// Clusters of 1 .. kMostSplit blocks that run at once on the device, asked once; only whether any does is of interest (choose).
struct Fit { int clusters[2][kMostSplit + 1]; };
template <int TN>
cudaError_t fill_fit(int (&clusters)[kMostSplit + 1]) {
    cudaError_t e = cudaFuncSetAttribute(weight_grad_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<TN>::total);
    for (int s = 1; s <= kMostSplit && e == cudaSuccess; ++s) {
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = s; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
        cudaLaunchConfig_t c = {};
        c.gridDim = s; c.blockDim = kThreads; c.dynamicSmemBytes = Layout<TN>::total; c.attrs = &at; c.numAttrs = 1;
        e = cudaOccupancyMaxActiveClusters(&clusters[s], weight_grad_kernel<TN>, &c);
    }
    return e;
}
cudaError_t device_fit(int dev, const Fit** out) {
    static std::mutex mu;
    static Fit fits[64];
    static bool done[64] = {false};
    std::lock_guard<std::mutex> lock(mu);
    if (!done[dev]) {
        cudaError_t e = fill_fit<128>(fits[dev].clusters[0]);
        if (e == cudaSuccess) e = fill_fit<256>(fits[dev].clusters[1]);
        if (e != cudaSuccess) return e;
        done[dev] = true;
    }
    *out = &fits[dev];
    return cudaSuccess;
}

int tiles_of(int cols, int D, int TN) { return (cols + kTM - 1) / kTM * ((D + TN - 1) / TN); }

// What bounds a block is what its SM can fetch (90 GB/s measured; the tensor cores would take twice that), so the tile width and the split
// are those with the least to fetch per block, rounds of clusters counted.  How many clusters run at once differs from one B200 to the next (148 SMs in
// GPCs of different sizes), but the split is the order of the sums, and a call has to return the same bits on every one: so the figures are
// those of one GPU (cudaOccupancyMaxActiveClusters for both widths), wherever this runs.
constexpr int kAtOnce[kMostSplit + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
struct Share { bool wide; int split; };
Share choose(const int* cols, int count, long long rows, int D) {
    Share best = {true, 1};
    long long least = -1;
    const long long blocks = (rows + kBox - 1) / kBox;
    for (int w = 1; w >= 0; --w) {
        int tiles = 0;
        for (int k = 0; k < count; ++k) tiles += tiles_of(cols[k], D, w ? 256 : 128);
        for (int s = 1; s <= kMostSplit && s <= blocks; ++s) {
            const int at_once = kAtOnce[s];
            // steps of 64 rows, and about five steps' worth of time to start and to add the tiles
            const long long cost = (long long)((tiles + at_once - 1) / at_once) * ((blocks + s - 1) / s + 5) * (w ? 3 : 2);
            if (least < 0 || cost < least) { least = cost; best = {w != 0, s}; }
        }
    }
    return best;
}

}  // namespace wgrad

cudaError_t read_wgrad_error(int* value, bool reset) {
    cudaError_t e = cudaMemcpyFromSymbol(value, stg::g_stage_error, sizeof(int));
    if (e == cudaSuccess && reset && *value != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(stg::g_stage_error, &zero, sizeof(int));
    }
    return e;
}

namespace wgrad {

template <int TN, bool STALL>
cudaError_t launch(const Args& a, int tiles, const CUtensorMap* maps, cudaStream_t s) {
    if (STALL)
        if (cudaError_t e = cudaFuncSetAttribute(weight_grad_kernel<TN, STALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<TN>::total)) return e;
    return launch_clusters_after(a.split, weight_grad_kernel<TN, STALL>, tiles * a.split, kThreads, Layout<TN>::total, s, a, maps[0], maps[1], maps[2], maps[3]);
}

bool bad_sizes(const int* cols, int count, long long rows, int D) {
    if (count < 1 || count > DSQG_WGRAD_MAX || rows < 1 || rows > (1LL << 30) || D < kBox || D % kBox || D > (1 << 20)) return true;
    for (int k = 0; k < count; ++k)
        if (cols[k] < kBox || cols[k] % kBox || cols[k] > (1 << 20)) return true;
    return false;
}

template <bool STALL>
int weight_grads(const void* const* dy, const long long* dy_stride, const int* cols, const void* const* x, float* const* dw, float* const* sums,
                 int count, long long rows, int D, long long limit, void* stream) {
    if (!dy || !dy_stride || !cols || !x || !dw || !sums) return DSQG_ERR_NULL_POINTER;
    if (bad_sizes(cols, count, rows, D)) return DSQG_ERR_BAD_SHAPE;
    if (!stg::tensor_map_encoder_available()) return DSQG_ERR_UNSUPPORTED;
    int dev = 0;
    const auto off16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return DSQG_ERR_CUDA;
    const Fit* fit = nullptr;
    if (device_fit(dev, &fit) != cudaSuccess) { cudaGetLastError(); return DSQG_ERR_CUDA; }
    Args a = {};
    CUtensorMap maps[2 * DSQG_WGRAD_MAX] = {};
    a.rows = (int)rows; a.D = D; a.limit = limit;
    for (int k = 0; k < count; ++k) {
        if (!dy[k] || !x[k] || !dw[k]) return DSQG_ERR_NULL_POINTER;
        if (off16(dy[k]) || off16(x[k]) || off16(dw[k]) || dy_stride[k] < cols[k] || dy_stride[k] % 8 || dy_stride[k] > (1 << 24)) return DSQG_ERR_MISALIGNED;
        a.job[k].cols = cols[k]; a.job[k].dw = dw[k]; a.job[k].sum = sums[k];
        // 64-column blocks of a row-major matrix as the "heads" of a tensor of 64-wide rows
        if (!stg::make_map(&maps[2 * k], &a.job[k].a_hf, dy[k], 1, cols[k] / kBox, (int)rows, kBox, rows * dy_stride[k], kBox, dy_stride[k], kBox) ||
            !stg::make_map(&maps[2 * k + 1], &a.job[k].b_hf, x[k], 1, D / kBox, (int)rows, kBox, rows * D, kBox, D, kBox))
            return DSQG_ERR_UNSUPPORTED;
    }
    if (count == 1) { maps[2] = maps[0]; maps[3] = maps[1]; }
    if (wait_error_seen()) return DSQG_ERR_WAIT;
    a.report = wait_error_word();
    const Share p = choose(cols, count, rows, D);
    if (fit->clusters[p.wide][p.split] < 1) return DSQG_ERR_UNSUPPORTED;       // part of a GPU that is too small for such a cluster
    a.split = p.split;
    int tiles = 0;
    for (int k = 0; k < count; ++k) a.job[k].tiles_end = tiles += tiles_of(a.job[k].cols, D, p.wide ? 256 : 128);
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    const cudaError_t e = p.wide ? launch<256, STALL>(a, tiles, maps, s) : launch<128, STALL>(a, tiles, maps, s);
    return e == cudaSuccess ? DSQG_OK : DSQG_ERR_CUDA;
}

}  // namespace wgrad
}  // namespace dsqg

extern "C" {

int dsqg_weight_grads_split(const int* cols, int count, long long rows, int D, int* tile_cols) {
    using namespace dsqg::wgrad;
    if (!cols || !tile_cols) return DSQG_ERR_NULL_POINTER;
    if (bad_sizes(cols, count, rows, D)) return DSQG_ERR_BAD_SHAPE;
    const Share p = choose(cols, count, rows, D);
    *tile_cols = p.wide ? 256 : 128;
    return p.split;
}

int dsqg_weight_grads(const void* const* dy, const long long* dy_stride, const int* cols, const void* const* x, float* const* dw, float* const* sums,
                      int count, long long rows, int D, void* stream) {
    return dsqg::wgrad::weight_grads<false>(dy, dy_stride, cols, x, dw, sums, count, rows, D, dsqg::wgrad::kLimit, stream);
}

int dsqg_test_weight_grads_timeout(const void* const* dy, const long long* dy_stride, const int* cols, const void* const* x, float* const* dw, float* const* sums,
                                   int count, long long rows, int D, long long limit_cycles, void* stream) {
    if (limit_cycles < 1 || limit_cycles > 2000000000LL) return DSQG_ERR_UNSUPPORTED;
    return dsqg::wgrad::weight_grads<true>(dy, dy_stride, cols, x, dw, sums, count, rows, D, limit_cycles, stream);
}

}  // extern "C"
