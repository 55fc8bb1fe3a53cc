// Warp-level building blocks of the tensor-core DSQG kernels (bf16, sm_100a).
//
// Fragment convention used by every kernel in dsqg_mma*.cu
// --------------------------------------------------------
// lane = 4*g + tig  (g = 0..7, tig = 0..3).  A warp owns a tile of 16 rows.
// A row of D bf16 elements is split into groups of 64, 32 and 16 elements (as many of each as fit, in this order); thread tig reads
// a quarter of every group: elements 64*c + 16*tig + [0,16), then 8*tig + [0,8) of a 32-element group, then 4*tig + [0,4) of
// a 16-element tail.
// Those D/4 elements are the thread's share of the contraction dimension for BOTH
// operands of  mma.sync.m16n8k16  (the instruction assigns k-indices {2tig,2tig+1,2tig+8,
// 2tig+9} of every k-step to thread tig in the A and in the B fragment alike, so any fixed
// assignment of physical d to k-index is legal as long as A and B agree).  Hence
//   * a "row fragment" (RowFrag) is loaded with one load per group,
//   * the same RowFrag serves as A operand (rows g, g+8 of the warp tile) or as B operand
//     (row g of an 8-row n-tile) of a product that contracts over d,
//   * movmatrix(.trans) turns a RowFrag into the B operand of a product that contracts over
//     ROWS (P.V, dS.K, ...); column n of n-tile j of such a product is element n&1 of register j of
//     thread n>>1, so thread tig ends up owning the elements of rows g and g+8 that it would load of
//     them: one store per group.
#pragma once

#include <type_traits>

#include "dsqg_common.cuh"

namespace dsqg {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kNeg = -1.0e30f;   // finite "minus infinity": masked scores
constexpr float kMinM = -1.0e29f;  // floor of the running row maximum: exp2(kNeg - kMinM) == 0

template <int D> struct RowFrag { uint32_t r[D / 8]; };
template <int D> constexpr bool kTail = D % 32 == 16;      // 8 bytes per thread
template <int D> constexpr bool kMid = D % 64 >= 32;       // 16 bytes per thread
template <int D> constexpr int kLane = D >= 64 ? 16 : 8;   // consecutive elements of a row a thread holds (of the first piece)

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Where the 16-byte and 8-byte pieces of a row lie from the thread's first piece on (row + kLane<D> * tig).
template <int D> __device__ __forceinline__ int mid_at() { return D >= 64 ? D / 64 * 64 - 8 * (int)(threadIdx.x & 3) : 0; }
template <int D> __device__ __forceinline__ int tail_at() { return D - 16 - (kLane<D> - 4) * (int)(threadIdx.x & 3); }

// p: this thread's first piece of the row (row + kLane<D> * tig).  64 elements are one load of 32 bytes per thread, so that the
// four lanes of a row cover a whole 128-byte line: the L1 takes a line per cycle whatever part of it is wanted, so 16-byte pieces
// (half a line per row and load) cost twice the passes.  B16 H12 N2048 D64: forward 104.8 -> 91.0, dQ 135.5 -> 122.0,
// dK/dV 157.5 -> 137.3 us.  A32 = false: pieces aligned to 16 bytes only.
template <int D, bool A32 = true>
__device__ __forceinline__ void load_row_at(RowFrag<D>& f, const __nv_bfloat16* p) {
#pragma unroll
    for (int c = 0; c < D / 64; ++c) {
        if constexpr (A32) {
            asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                : "=r"(f.r[8 * c]), "=r"(f.r[8 * c + 1]), "=r"(f.r[8 * c + 2]), "=r"(f.r[8 * c + 3]), "=r"(f.r[8 * c + 4]),
                  "=r"(f.r[8 * c + 5]), "=r"(f.r[8 * c + 6]), "=r"(f.r[8 * c + 7]) : "l"(p + 64 * c));
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 u = __ldg(reinterpret_cast<const uint4*>(p + 64 * c) + h);
                f.r[8 * c + 4 * h] = u.x; f.r[8 * c + 4 * h + 1] = u.y; f.r[8 * c + 4 * h + 2] = u.z; f.r[8 * c + 4 * h + 3] = u.w;
            }
        }
    }
    if constexpr (kMid<D>) {
        constexpr int J = D / 64 * 8;
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(p + mid_at<D>()));
        f.r[J] = u.x; f.r[J + 1] = u.y; f.r[J + 2] = u.z; f.r[J + 3] = u.w;
    }
    if constexpr (kTail<D>) {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(p + tail_at<D>()));
        f.r[D / 8 - 2] = u.x; f.r[D / 8 - 1] = u.y;
    }
}

// This thread's pieces from p on, zero when !valid (the pointer is not dereferenced then).
template <int D, bool A32 = true>
__device__ __forceinline__ void load_piece(RowFrag<D>& f, const __nv_bfloat16* p, bool valid) {
#pragma unroll
    for (int j = 0; j < D / 8; ++j) f.r[j] = 0u;
    if (valid) load_row_at<D, A32>(f, p);
}
// One row; zero-filled when !valid.
template <int D, bool A32 = true>
__device__ __forceinline__ void load_row(RowFrag<D>& f, const __nv_bfloat16* row_ptr, int tig, bool valid) {
#pragma unroll
    for (int j = 0; j < D / 8; ++j) f.r[j] = 0u;
    if (valid) load_row_at<D, A32>(f, row_ptr + kLane<D> * tig);
}

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// d = A.B with a zero accumulator input (no register initialisation needed)
__device__ __forceinline__ void mma16816_z(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                           uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// c = A.B (overwrites c), contraction over d as in mma_rows
template <int D>
__device__ __forceinline__ void mma_rows_z(float (&c)[4], const RowFrag<D>& a_lo, const RowFrag<D>& a_hi,
                                           const RowFrag<D>& b) {
    mma16816_z(c, a_lo.r[0], a_hi.r[0], a_lo.r[1], a_hi.r[1], b.r[0], b.r[1]);
#pragma unroll
    for (int kk = 1; kk < D / 16; ++kk)
        mma16816(c, a_lo.r[2 * kk], a_hi.r[2 * kk], a_lo.r[2 * kk + 1], a_hi.r[2 * kk + 1], b.r[2 * kk], b.r[2 * kk + 1]);
}

// C[16 x 8] += A(rows g / g+8 = a_lo / a_hi)[16 x D] . B(row g = b)[8 x D]^T   (contracts over d)
template <int D>
__device__ __forceinline__ void mma_rows(float (&c)[4], const RowFrag<D>& a_lo, const RowFrag<D>& a_hi,
                                         const RowFrag<D>& b) {
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
        mma16816(c, a_lo.r[2 * kk], a_hi.r[2 * kk], a_lo.r[2 * kk + 1], a_hi.r[2 * kk + 1], b.r[2 * kk], b.r[2 * kk + 1]);
}

__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}

template <int D>
__device__ __forceinline__ void transpose_frag(RowFrag<D>& t, const RowFrag<D>& f) {
#pragma unroll
    for (int j = 0; j < D / 8; ++j) t.r[j] = movmatrix_trans(f.r[j]);
}

// acc[16 x D] += A[16 x 16] . B[16 x D]  where the 16 contraction rows are the rows of the two
// transposed row fragments (rows 0..7 = t_lo, rows 8..15 = t_hi).  acc[j] is n-tile j.
template <int D>
__device__ __forceinline__ void mma_cols(float (&acc)[D / 8][4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         const RowFrag<D>& t_lo, const RowFrag<D>& t_hi) {
#pragma unroll
    for (int j = 0; j < D / 8; ++j) mma16816(acc[j], a0, a1, a2, a3, t_lo.r[j], t_hi.r[j]);
}

__device__ __forceinline__ float quad_max(float x) {
    x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
    return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
}
__device__ __forceinline__ float quad_sum(float x) {
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x + __shfl_xor_sync(0xffffffffu, x, 2);
}

// Diagonal A fragment: A[g][g] = x_lo, A[g+8][g+8] = x_hi, zero elsewhere.  Only the thread
// with tig == g>>1 holds non-zeros (element g&1 of its a0a1 / a6a7 registers).
__device__ __forceinline__ void diag_frag(float x_lo, float x_hi, bool owner, int g, uint32_t& a0, uint32_t& a3) {
    const uint32_t lo = owner ? (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x_lo)) : 0u;
    const uint32_t hi = owner ? (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x_hi)) : 0u;
    const int sh = (g & 1) * 16;
    a0 = lo << sh;
    a3 = hi << sh;
}

// Store rows g and g+8 of an accumulator tile (the elements of load_row_at) as bf16, scaled per row.
template <int D, bool A32>
__device__ __forceinline__ void store_row_at(const uint32_t (&w)[D / 8], __nv_bfloat16* p) {
#pragma unroll
    for (int c = 0; c < D / 64; ++c) {
        if constexpr (A32) {
            asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" :: "l"(p + 64 * c), "r"(w[8 * c]), "r"(w[8 * c + 1]), "r"(w[8 * c + 2]),
                         "r"(w[8 * c + 3]), "r"(w[8 * c + 4]), "r"(w[8 * c + 5]), "r"(w[8 * c + 6]), "r"(w[8 * c + 7]) : "memory");
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *(reinterpret_cast<uint4*>(p + 64 * c) + h) = make_uint4(w[8 * c + 4 * h], w[8 * c + 4 * h + 1], w[8 * c + 4 * h + 2], w[8 * c + 4 * h + 3]);
        }
    }
    if constexpr (kMid<D>) {
        constexpr int J = D / 64 * 8;
        *reinterpret_cast<uint4*>(p + mid_at<D>()) = make_uint4(w[J], w[J + 1], w[J + 2], w[J + 3]);
    }
    if constexpr (kTail<D>) *reinterpret_cast<uint2*>(p + tail_at<D>()) = make_uint2(w[D / 8 - 2], w[D / 8 - 1]);
}
template <int D, bool A32 = true>
__device__ __forceinline__ void store_acc_rows(const float (&acc)[D / 8][4], __nv_bfloat16* row_lo, __nv_bfloat16* row_hi,
                                               bool ok_lo, bool ok_hi, float s_lo, float s_hi, int tig) {
    uint32_t w[D / 8];
#pragma unroll
    for (int j = 0; j < D / 8; ++j) w[j] = pack_bf16x2(acc[j][0] * s_lo, acc[j][1] * s_lo);
    if (ok_lo) store_row_at<D, A32>(w, row_lo + kLane<D> * tig);
#pragma unroll
    for (int j = 0; j < D / 8; ++j) w[j] = pack_bf16x2(acc[j][2] * s_hi, acc[j][3] * s_hi);
    if (ok_hi) store_row_at<D, A32>(w, row_hi + kLane<D> * tig);
}

// As store_acc_rows, with every element multiplied by sigmoid(gate) of the same position (gate rows
// are bf16 in the layout of the output rows): the sigmoid gate of the attention block folded into
// the epilogue (DWARF train/train_2048_condU.py:190-191).
template <int D, bool A32 = true>
__device__ __forceinline__ void store_acc_rows_gated(const float (&acc)[D / 8][4], __nv_bfloat16* row_lo, __nv_bfloat16* row_hi,
                                                     const __nv_bfloat16* gate_lo, const __nv_bfloat16* gate_hi,
                                                     bool ok_lo, bool ok_hi, float s_lo, float s_hi, int tig) {
    auto sig2 = [](uint32_t u, float& a, float& b) {
        a = __fdividef(1.f, 1.f + __expf(-__uint_as_float(u << 16)));
        b = __fdividef(1.f, 1.f + __expf(-__uint_as_float(u & 0xffff0000u)));
    };
    auto half = [&](auto HC, const __nv_bfloat16* gate, __nv_bfloat16* row, float s) {
        constexpr int H = decltype(HC)::value;
        RowFrag<D> gf;
        load_row_at<D, A32>(gf, gate + kLane<D> * tig);
        uint32_t w[D / 8];
#pragma unroll
        for (int j = 0; j < D / 8; ++j) {
            float a, b;
            sig2(gf.r[j], a, b);
            w[j] = pack_bf16x2(acc[j][2 * H] * s * a, acc[j][2 * H + 1] * s * b);
        }
        store_row_at<D, A32>(w, row + kLane<D> * tig);
    };
    if (ok_lo) half(std::integral_constant<int, 0>(), gate_lo, row_lo, s_lo);
    if (ok_hi) half(std::integral_constant<int, 1>(), gate_hi, row_hi, s_hi);
}

// One row of the sigmoid gate's backward (this thread's elements): d is dy and becomes dout = dy * s, y becomes dgate = dy * y * (1 - s), s = sigmoid(gate).
template <int D>
__device__ __forceinline__ void gate_row(RowFrag<D>& d, RowFrag<D>& y, const RowFrag<D>& gate) {
#pragma unroll
    for (int j = 0; j < D / 8; ++j) {
        float out[2], dg[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            auto f = [&](uint32_t u) { return __uint_as_float(i ? u & 0xffff0000u : u << 16); };
            const float s = __fdividef(1.f, 1.f + __expf(-f(gate.r[j]))), dy = f(d.r[j]);
            out[i] = dy * s;
            dg[i] = dy * f(y.r[j]) * (1.f - s);
        }
        d.r[j] = pack_bf16x2(out[0], out[1]);
        y.r[j] = pack_bf16x2(dg[0], dg[1]);
    }
}

// Partial dot product of two row fragments over this thread's elements (fp32).
template <int D>
__device__ __forceinline__ float frag_dot(const RowFrag<D>& a, const RowFrag<D>& b) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < D / 8; ++j) {
        s = fmaf(__uint_as_float(a.r[j] << 16), __uint_as_float(b.r[j] << 16), s);
        s = fmaf(__uint_as_float(a.r[j] & 0xffff0000u), __uint_as_float(b.r[j] & 0xffff0000u), s);
    }
    return s;
}

// The whole row's dot product on all four lanes.  At D = 32 its elements are added one after the other, as one thread would: ds = P (dP - delta) is
// rounded to bf16, and another order moves single roundings, which a gradient that nearly cancels (a bias on every key) shows.
template <int D>
__device__ __forceinline__ float row_dot(const RowFrag<D>& a, const RowFrag<D>& b) {
    if constexpr (D == 32) {
        float acc = 0.f;
#pragma unroll
        for (int l = 0; l < 4; ++l) {                        // every lane adds its products to what the lane before has; the l-th lane's count
            float s = l ? __shfl_sync(0xffffffffu, acc, l - 1, 4) : 0.f;
#pragma unroll
            for (int j = 0; j < D / 8; ++j) {
                s = fmaf(__uint_as_float(a.r[j] << 16), __uint_as_float(b.r[j] << 16), s);
                s = fmaf(__uint_as_float(a.r[j] & 0xffff0000u), __uint_as_float(b.r[j] & 0xffff0000u), s);
            }
            acc = s;
        }
        return __shfl_sync(0xffffffffu, acc, 3, 4);
    } else {
        return quad_sum(frag_dot(a, b));
    }
}

// Lane roles inside a 16-row tile held as MMA fragments (rows g and g+8 per lane).
struct Lane {
    int warp, lane, g, tig;
    bool owner;          // holds the diagonal entries of rows g and g+8
    int owner_lane;      // lane of this quad's owner
    __device__ Lane() {
        warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); lane = threadIdx.x & 31; g = lane >> 2; tig = lane & 3;
        owner = tig == (g >> 1);
        owner_lane = (lane & ~3) | (g >> 1);
    }
};

// acc(rows g / g+8) += x_lo * f_lo, x_hi * f_hi for this thread's elements: the diagonal form of
// "A.B with A = diag(x)" -- row g of the product only needs row g of B, which the thread holds
// as a row fragment for exactly the elements d its accumulators cover.
template <int D>
__device__ __forceinline__ void diag_fma(float (&acc)[D / 8][4], float x_lo, float x_hi, const RowFrag<D>& f_lo,
                                         const RowFrag<D>& f_hi) {
    // packed fp32 FMA (fma.rn.f32x2, sm_100): one instruction updates the two accumulators a row has
    // in an n-tile; measured 1 % off the step against scalar FMAs (cfg1: 284.8 against 287.6 us)
    unsigned long long xl, xh;
    asm("mov.b64 %0, {%1, %1};" : "=l"(xl) : "f"(x_lo));
    asm("mov.b64 %0, {%1, %1};" : "=l"(xh) : "f"(x_hi));
#pragma unroll
    for (int j = 0; j < D / 8; ++j) {
        const uint32_t u0 = f_lo.r[j], u1 = f_hi.r[j];
        unsigned long long v0, v1, c0, c1;
        asm("mov.b64 %0, {%1, %2};" : "=l"(v0) : "r"(u0 << 16), "r"(u0 & 0xffff0000u));
        asm("mov.b64 %0, {%1, %2};" : "=l"(v1) : "r"(u1 << 16), "r"(u1 & 0xffff0000u));
        asm("mov.b64 %0, {%1, %2};" : "=l"(c0) : "f"(acc[j][0]), "f"(acc[j][1]));
        asm("mov.b64 %0, {%1, %2};" : "=l"(c1) : "f"(acc[j][2]), "f"(acc[j][3]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c0) : "l"(xl), "l"(v0));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c1) : "l"(xh), "l"(v1));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[j][0]), "=f"(acc[j][1]) : "l"(c0));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[j][2]), "=f"(acc[j][3]) : "l"(c1));
    }
}

// The running maximum of the online softmax only moves when a score exceeds it by more than this
// (log2 units): probabilities stay below 2^kSlack, which fp32 sums and bf16 values absorb.
constexpr float kSlack = 16.f;

}  // namespace dsqg
