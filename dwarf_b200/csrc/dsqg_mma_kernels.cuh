// Tensor-core DSQG kernels (bf16 storage, fp32 accumulate) for D in {32, 64} (dense windows up
// to 64 wide) and D in {48, 80, 96, 128} (dense windows up to 32 wide; 48 and 80 contiguous tensors without
// scale_embed only).
//
// One warp owns 16 consecutive rows of one (batch, head) sequence.  The dense window is a
// banded GEMM: the 16 query rows against the WB+16 key rows [g0-WB, g0+16) with
// mma.sync.m16n8k16; out-of-band entries are masked.  Every sparse tap pairs row n with row
// n-delta, i.e. it is the diagonal of a 16x16 tile: its scores come from two m16n8 MMAs per
// k-step, of which the thread with tig == g>>1 keeps the diagonal entries; the products that
// follow (p.v, ds.k, ds.q, p.dO) scale row g of a tile the thread already holds as a row
// fragment, so they are plain fp32 FMAs on the thread's accumulators (no transposes, no tensor
// core: measured faster than a diagonal A fragment).  The math is that of the DWARF reference kernels
// (kernels/dsqg_attention_v3.py:60-163 forward, :198-275 dQ, :282-352 dK/dV), with the per-head
// output gain of train/train_2048_condU.py:187 fused in.  See dsqg_mma.cuh for the fragment
// conventions.  scale_embed (D <= 64): q.scale_embed[j] is computed per 16-row tile with
// split-bf16 MMAs into a shared-memory tile that also carries the position bias and replaces
// the start-value table; the dQ kernel adds dS.scale_embed (MMA, dS from its staging tile),
// produces dscale_embed partials per 64-row tile (dS^T.Q, MMA; dse_group_kernel adds groups of
// eight tiles) and leaves the per-row tile in global memory for the dK/dV kernel.
#pragma once

#include "dsqg_mma.cuh"
#include <initializer_list>
#include <mutex>
#include <type_traits>

namespace dsqg {
namespace {

constexpr int kWarps = 4;
constexpr int kRows = 16 * kWarps; // rows per CTA

// How q, k, v, out, ... are addressed: contiguous [B,H,N,D]; through the element strides in FwdArgs / BwdArgs (rows of D
// contiguous elements; any batch / head / row strides), e.g. the un-permuted output of a fused qkv projection and a token-major
// result; the same with pieces that are aligned to 16 bytes only where a piece is 32 (D >= 64); backward only: strides for the
// gradients, everything that is read contiguous.
constexpr int kContiguous = 0, kStrided = 1, kStridedAny = 2, kKept = 3;

// Where this thread's piece of row `tile row + g + rows` of a tensor lies: a pointer that is the same for the whole warp, plus a lane part (32 bits where
// rows follow one another, CI).  A tap's address is then formed once per warp by the uniform datapath, and K and V share the lane part;
// a pointer per lane and tensor cost four more registers and four vector instructions per tap and tensor, which these kernels, held to the
// registers of four to six CTAs per SM, paid for in spills.  The product is opaque, or the compiler adds the lane part first.
template <int D, bool CI> struct Rows {
    const __nv_bfloat16* tile;
    long long rs;                                        // row stride in bytes (strided tensors)
    std::conditional_t<CI, unsigned, long long> lane;
    // p: row 0 of the sequence; row0: first row of the tile; stride: elements from row to row
    __device__ __forceinline__ Rows(const void* p, size_t base, int row0, ptrdiff_t stride, const Lane& L) {
        tile = static_cast<const __nv_bfloat16*>(p) + base + (ptrdiff_t)row0 * stride;
        rs = 2 * (long long)stride;
        if constexpr (CI) lane = 2u * (unsigned)(L.g * D + kLane<D> * L.tig);
        else lane = L.g * rs + 2 * kLane<D> * L.tig;
    }
    __device__ __forceinline__ const __nv_bfloat16* at(int rows) const {
        unsigned long long x;
        if constexpr (CI) asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(x) : "r"(rows), "n"(2 * D), "l"(tile));
        else asm("mad.lo.s64 %0, %1, %2, %3;" : "=l"(x) : "l"((long long)rows), "l"(rs), "l"(tile));
        return reinterpret_cast<const __nv_bfloat16*>(x + lane);
    }
    // rows r and r + 8
    template <bool AL> __device__ __forceinline__ void load2(RowFrag<D>& lo, RowFrag<D>& hi, int rows) const {
        const __nv_bfloat16* x = at(rows);
        load_row_at<D, AL>(lo, x);
        load_row_at<D, AL>(hi, CI ? x + 8 * D : at(rows + 8));
    }
    template <bool AL> __device__ __forceinline__ void load2(RowFrag<D>& lo, RowFrag<D>& hi, int rows, bool v_lo, bool v_hi) const {
        const __nv_bfloat16* x = at(rows);
        load_piece<D, AL>(lo, x, v_lo);
        load_piece<D, AL>(hi, CI ? x + 8 * D : at(rows + 8), v_hi);
    }
};

// ------------------------------------------------------------------------------ forward
// Online softmax over the dense window, then over the sparse taps, with the per-element
// bookkeeping moved out of the tile loop:
//   * the band mask and the position bias of the dense window are the INITIAL VALUE of the score
//     accumulators (two 8-byte loads per n-tile from a table over the offsets, StartTable), so the
//     scores leave the MMAs already biased and masked (in units of 1/scale);
//   * interior tiles (all band rows inside the sequence) load with no predicates and constant
//     offsets from one pointer; a sparse tap whose 16 key rows all exist does the same;
//   * the running maximum only moves when a sparse score exceeds it by more than kSlack
//     (log2 units): p stays below 2^kSlack, which fp32 sums and bf16 probabilities absorb;
//   * lanes that do not own a diagonal entry subtract +1e30 instead of the maximum, so their
//     probability is exactly zero without a select.
// Scale embedding: s_j += q.scale_embed[j] / sqrt(D) (reference: kernels/dsqg_attention_v3.py:112-118).  q.scale_embed is formed
// per 16-row tile with MMAs, in the order the scores need it: column x = WB + 16 - delta for the dense offsets (as StartTable), then
// the sparse taps.  Row i of a tile reads its start values at x = 16 - i + c, pairs of them 8-byte aligned (the row
// pitch is odd and 9 mod 32: no bank conflicts), at compile-time distances from one address per lane.  The earlier tiles in tap
// order were gathered through a table of offsets: an index load, four address computations and four loads per n-tile.
//   hi + lo: bf16 halves of the table rows (their sum carries 16 mantissa bits), kDense rows for x = 16 .. WB + 23, then
//   the sparse taps rounded up to eight; pb: pos_bias / scale per row, the mask value where the row is no tap.
template <int WB> struct SeGeo {
    static constexpr int kC = WB + 16, kTiles = WB / 8 + 1, kDense = 8 * kTiles, kPitch = WB == 32 ? 73 : 105;
    static __host__ __device__ int rows(int ns) { return kDense + (ns + 7) / 8 * 8; }
    static __host__ __device__ int sparse_pitch(int ns) { return (ns + 7) / 8 * 8 + 1; }
    // tap of table row r, -1: none
    static __device__ __forceinline__ int tap(const Taps& t, int r) {
        const int j = r < kDense ? WB - r - t.d_lo : t.n_dense + r - kDense;
        return r < kDense ? (j >= 0 && j < t.n_dense ? j : -1) : (j < t.J ? j : -1);
    }
};
struct SeRows { const __nv_bfloat16* hi; const __nv_bfloat16* lo; const float* pb; };

// The tile of 16 query rows (A fragments qa: rows g, qb: rows g + 8): dense part to dense[row * pitch + x], sparse part to
// sparse[row * sp + tap], and to rows_lo / rows_hi (nullable, global memory).  GL: the table is in global memory.
template <int D, int WB, bool GL>
__device__ __forceinline__ void build_se_tile(const SeRows& tab, int ns, const RowFrag<D>& qa, const RowFrag<D>& qb, int g, int tig, float* dense,
                                              int pitch, float* sparse, int sp, float* rows_lo = nullptr, float* rows_hi = nullptr) {
    using G = SeGeo<WB>;
    auto product = [&](int m, float (&c)[4]) {
        const float2* pbp = reinterpret_cast<const float2*>(tab.pb + 8 * m + 2 * tig);
        const float2 pb = GL ? __ldg(pbp) : *pbp;
        c[0] = c[2] = pb.x; c[1] = c[3] = pb.y;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            RowFrag<D> sf;
            const uint4* src = reinterpret_cast<const uint4*>((half ? tab.lo : tab.hi) + (8 * m + g) * D + kLane<D> * tig);
#pragma unroll
            for (int cc = 0; cc < D / 32; ++cc) {
                const int o = kLane<D> == 16 ? 8 * (cc >> 1) + (cc & 1) : 4 * cc;
                const uint4 u = GL ? __ldg(src + o) : src[o];
                sf.r[4 * cc + 0] = u.x; sf.r[4 * cc + 1] = u.y; sf.r[4 * cc + 2] = u.z; sf.r[4 * cc + 3] = u.w;
            }
            mma_rows(c, qa, qb, sf);
        }
    };
    float* at = dense + g * pitch + 16 + 2 * tig;
#pragma unroll
    for (int m = 0; m < G::kTiles; ++m) {
        float c[4];
        product(m, c);
        at[8 * m] = c[0]; at[8 * m + 1] = c[1];
        at[8 * pitch + 8 * m] = c[2]; at[8 * pitch + 8 * m + 1] = c[3];
    }
    at = sparse + g * sp + 2 * tig;
#pragma unroll 1
    for (int m = 0; 8 * m < ns; ++m) {
        float c[4];
        product(G::kTiles + m, c);
        at[8 * m] = c[0]; at[8 * m + 1] = c[1];
        at[8 * sp + 8 * m] = c[2]; at[8 * sp + 8 * m + 1] = c[3];
        if (rows_lo) *reinterpret_cast<float2*>(rows_lo + 8 * m + 2 * tig) = make_float2(c[0], c[1]);
        if (rows_hi) *reinterpret_cast<float2*>(rows_hi + 8 * m + 2 * tig) = make_float2(c[2], c[3]);
    }
    __syncwarp();
}
// Start values of n-tile nt; lane: dense + g * pitch + 16 - g + 2 tig.  Columns below x = 16 and from WB + 24 on are not in the tile:
// they belong to no offset.
template <int WB>
__device__ __forceinline__ void se_start(float (&s)[4], const float* lane, int pitch, int nt, int g, int tig) {
    const int c = 2 * tig;
    const float2 lo = *reinterpret_cast<const float2*>(lane + 8 * nt);
    s[0] = lo.x; s[1] = lo.y; s[2] = s[3] = kNeg;
    if (nt > 0) {
        const float2 hi = *reinterpret_cast<const float2*>(lane + 8 * (pitch - 1) + 8 * nt);
        s[2] = hi.x; s[3] = hi.y;
    }
    if (nt == 0) { if (c < g) s[0] = kNeg; if (c + 1 < g) s[1] = kNeg; }
    if (nt == 1) { if (c < g) s[2] = kNeg; if (c + 1 < g) s[3] = kNeg; }
    if (nt == WB / 8 + 1) { if (c >= g) s[0] = kNeg; if (c + 1 >= g) s[1] = kNeg; }
}

// The table in shared memory (all threads of the CTA; the caller syncs): hi | lo | pb, then what follows it.
template <int D, int WB, int THREADS>
__device__ __forceinline__ SeRows fill_se_rows(float* smem, const float* scale_embed, const float* pos_bias, const Taps& t, int H, int h, float scale) {
    const int R = SeGeo<WB>::rows(t.n_sparse);
    __nv_bfloat16* hi = reinterpret_cast<__nv_bfloat16*>(smem);
    __nv_bfloat16* lo = hi + R * D;
    float* pb = reinterpret_cast<float*>(lo + R * D);
    for (int e = threadIdx.x; e < R * (D / 4); e += THREADS) {
        const int j = SeGeo<WB>::tap(t, e / (D / 4));
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j >= 0) x = __ldg(reinterpret_cast<const float4*>(scale_embed + j * D) + e % (D / 4));
        const __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
        reinterpret_cast<uint2*>(hi)[e] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        reinterpret_cast<uint2*>(lo)[e] = make_uint2(pack_bf16x2(x.x - __low2float(a), x.y - __high2float(a)),
                                                     pack_bf16x2(x.z - __low2float(b), x.w - __high2float(b)));
    }
    const float inv_scale = 1.f / scale;
    for (int r = threadIdx.x; r < R; r += THREADS) {
        const int j = SeGeo<WB>::tap(t, r);
        pb[r] = j >= 0 ? pos_bias[j * H + h] * inv_scale : kNeg;
    }
    return {hi, lo, pb};
}
// The same for the backward, where rows are keys (dK/dV) and the tile holds the query rows of the whole CTA: element (key i, query c)
// of a warp's tile belongs to row c, column WB + 16 - c + i.  lane: tile of the warp's first query + 2 tig (pitch - 1) + WB + 16 + g; the
// pitch is 5 mod 32, so that the eight keys of four queries hit different banks.
template <int WB> constexpr int kSeKeyPitch = WB == 32 ? 69 : 101;
template <int WB>
__device__ __forceinline__ void se_start_keys(float (&s)[4], const float* lane, int nt, int g, int tig) {
    constexpr int Q = kSeKeyPitch<WB> - 1, last = WB / 8 + 1;
    const float* p = lane + 8 * nt * Q;
    const int c = 2 * tig;
    s[0] = p[0]; s[1] = p[Q]; s[2] = p[8]; s[3] = p[Q + 8];
    if (nt == last) { s[0] = s[1] = kNeg; if (g < c) s[2] = kNeg; if (g < c + 1) s[3] = kNeg; }
    if (nt == last - 1) { if (g < c) s[0] = kNeg; if (g < c + 1) s[1] = kNeg; }
    if (nt == 0) { if (g >= c) s[2] = kNeg; if (g >= c + 1) s[3] = kNeg; }
}

template <int WB> __host__ __device__ inline size_t se_rows_bytes(int ns, int D) { return (size_t)SeGeo<WB>::rows(ns) * (4 * D + 4); }
template <int WB> __host__ __device__ inline size_t se_tile_floats(int ns) { return (size_t)16 * (SeGeo<WB>::kPitch + SeGeo<WB>::sparse_pitch(ns)); }

// Start values of the score accumulators of the dense window.  Element (i, c) of a tile belongs to one offset
// (forward, dQ: WB + i - c; dK/dV: c - i), so the tile's values are a table over x = 16 - i + c, and the two
// columns of an accumulator pair are neighbours in it.  A second copy an odd distance away keeps the pair 8-byte
// aligned for odd rows, 16 banks from the first so that a half warp's loads do not collide.  146 floats for WB = 32
// against the 3 KB of a table per lane, which every 64-row block had to fill: about 100 instructions per 16-row tile
// and most of the time before the first load of K.  B32 H8 N2048 D32: forward 67.9 -> 65.0 us; D = 64, N = 4096: dQ 299 -> 287 us
// (with the staging of DsStage).
template <int WB> struct StartTable {
    static constexpr int kOdd = WB <= 48 ? 81 : 113, kSize = kOdd + WB + 33;
    // KEYS: rows are keys (dK/dV)
    template <bool KEYS, int THREADS>
    static __device__ __forceinline__ void fill(float* tab, const float* pos_bias, int H, int h, int d_lo, int d_hi, float scale) {
        const float inv_scale = 1.f / scale;
        for (int e = threadIdx.x; e < kSize; e += THREADS) {
            const int x = e < kOdd ? e : e - kOdd, delta = KEYS ? x - 16 : WB + 16 - x;
            tab[e] = delta >= d_lo && delta <= d_hi ? pos_bias[(delta - d_lo) * H + h] * inv_scale : kNeg;
        }
    }
    // this lane's pointer: values of (g, 8 nt + 2 tig), (g, .. + 1) at [8 nt], of row g + 8 at [8 nt - 8]
    static __device__ __forceinline__ const float* lane(const float* tab, const Lane& L) { return tab + (L.g & 1) * kOdd + 16 - L.g + 2 * L.tig; }
    static __device__ __forceinline__ void get(float (&s)[4], const float* lane_tab, int nt) {
        const float2 lo = *reinterpret_cast<const float2*>(lane_tab + 8 * nt), hi = *reinterpret_cast<const float2*>(lane_tab + 8 * nt - 8);
        s[0] = lo.x; s[1] = lo.y; s[2] = hi.x; s[3] = hi.y;
    }
};

template <int D, int WB, bool INTERIOR, int kTapGroup, bool SE, int ST>
__device__ __forceinline__ void fwd_tile(const FwdArgs& a, const float* start, const int2* tap_s, const Taps& t, int ns,
                                         int bh, int h, int g0, const Lane& L, const SeRows& se, float* se_tile) {
    // scale_embed: the warp's tile, dense part first; qs0 / qs1: sparse entries of rows g / g + 8
    const int sp = SE ? SeGeo<WB>::sparse_pitch(ns) : 0;
    float* se_sparse = se_tile + 16 * SeGeo<WB>::kPitch;
    const float* qs0 = se_sparse + L.g * sp;
    const float* qs1 = qs0 + 8 * sp;
    constexpr int NT = (WB + 16) / 8;
    const int N = a.N, g = L.g, tig = L.tig;
    const int row_lo = g0 + g, row_hi = row_lo + 8;
    const bool ok_lo = INTERIOR || row_lo < N, ok_hi = INTERIOR || row_hi < N;
    constexpr bool AL = ST != kStridedAny;
    const ptrdiff_t RS = ST ? (ptrdiff_t)a.in_sn : D, OS = ST ? (ptrdiff_t)a.out_sn : D;   // row strides of q/k/v and of out
    const size_t base = ST ? (size_t)(bh / a.H) * a.in_sb + (size_t)h * a.in_sh : (size_t)bh * N * D;
    const size_t obase = ST ? (size_t)(bh / a.H) * a.out_sb + (size_t)h * a.out_sh : base;
    const Rows<D, !ST> qr(a.q, base, g0, RS, L), kr(a.k, base, g0, RS, L), vr(a.v, base, g0, RS, L);
    const float c2 = a.scale * kLog2e;
    const int kb0 = g0 - WB;

    RowFrag<D> qa, qb;
    qr.template load2<AL>(qa, qb, 0, ok_lo, ok_hi);
    // Copies for the backward: tensor x (0: q, 1: k, 2: v), rows g / g + 8
    auto keep = [&](int x, const RowFrag<D>& f, int row, bool ok) {
        if (ST && a.keep && ok)
            store_row_at<D, true>(f.r, static_cast<__nv_bfloat16*>(a.keep) + (((size_t)x * a.B * a.H + bh) * N + row) * D + kLane<D> * tig);
    };
    keep(0, qa, row_lo, ok_lo); keep(0, qb, row_hi, ok_hi);
    if constexpr (SE) build_se_tile<D, WB, false>(se, ns, qa, qb, g, tig, se_tile, SeGeo<WB>::kPitch, se_sparse, sp);
    const float* se_lane = se_tile + g * (SeGeo<WB>::kPitch - 1) + 16 + 2 * tig;

    // ---- dense window: key row of n-tile nt for this thread is kb0 + 8 nt + g = row_lo - WB + 8 nt
    const __nv_bfloat16* k_band = kr.at(-WB);
    float S[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        if constexpr (SE) {
            se_start<WB>(S[nt], se_lane, SeGeo<WB>::kPitch, nt, g, tig);
        } else {
            StartTable<WB>::get(S[nt], start, nt);
        }
        RowFrag<D> kf;
        const __nv_bfloat16* kp = ST ? kr.at(8 * nt - WB) : k_band + 8 * nt * D;
        if (INTERIOR) load_row_at<D, AL>(kf, kp);
        else load_piece<D, AL>(kf, kp, kb0 + 8 * nt + g >= 0 && kb0 + 8 * nt + g < N);
        if (nt >= WB / 8) keep(1, kf, nt == WB / 8 ? row_lo : row_hi, nt == WB / 8 ? ok_lo : ok_hi);
        mma_rows(S[nt], qa, qb, kf);
    }
    if (!INTERIOR && kb0 < 0) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (kb0 + 8 * nt + 2 * tig + (r & 1) < 0) S[nt][r] = kNeg;
    }
    float m_lo = kMinM, m_hi = kMinM;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        m_lo = fmaxf(m_lo, fmaxf(S[nt][0], S[nt][1]));
        m_hi = fmaxf(m_hi, fmaxf(S[nt][2], S[nt][3]));
    }
    m_lo = quad_max(m_lo) * c2; m_hi = quad_max(m_hi) * c2;          // log2 units from here on
    float l_lo = 0.f, l_hi = 0.f;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        S[nt][0] = ex2(fmaf(S[nt][0], c2, -m_lo)); S[nt][1] = ex2(fmaf(S[nt][1], c2, -m_lo));
        S[nt][2] = ex2(fmaf(S[nt][2], c2, -m_hi)); S[nt][3] = ex2(fmaf(S[nt][3], c2, -m_hi));
        l_lo += S[nt][0] + S[nt][1]; l_hi += S[nt][2] + S[nt][3];
    }
    float O[D / 8][4];
    const __nv_bfloat16* v_band = vr.at(-WB);
#pragma unroll
    for (int c = 0; c < NT / 2; ++c) {
        RowFrag<D> vf0, vf1, vt0, vt1;
        const __nv_bfloat16* vp0 = ST ? vr.at(16 * c - WB) : v_band + 16 * c * D;
        const __nv_bfloat16* vp1 = ST ? vr.at(16 * c + 8 - WB) : vp0 + 8 * D;
        if (INTERIOR) {
            load_row_at<D, AL>(vf0, vp0);
            load_row_at<D, AL>(vf1, vp1);
        } else {
            const int r = kb0 + 16 * c + g;
            load_piece<D, AL>(vf0, vp0, r >= 0 && r < N);
            load_piece<D, AL>(vf1, vp1, r + 8 >= 0 && r + 8 < N);
        }
        if (c == WB / 16) { keep(2, vf0, row_lo, ok_lo); keep(2, vf1, row_hi, ok_hi); }
        transpose_frag(vt0, vf0); transpose_frag(vt1, vf1);
        const uint32_t a0 = pack_bf16x2(S[2 * c][0], S[2 * c][1]), a1 = pack_bf16x2(S[2 * c][2], S[2 * c][3]);
        const uint32_t a2 = pack_bf16x2(S[2 * c + 1][0], S[2 * c + 1][1]), a3 = pack_bf16x2(S[2 * c + 1][2], S[2 * c + 1][3]);
        if (c == 0) {
#pragma unroll
            for (int j = 0; j < D / 8; ++j) mma16816_z(O[j], a0, a1, a2, a3, vt0.r[j], vt1.r[j]);
        } else {
            mma_cols<D>(O, a0, a1, a2, a3, vt0, vt1);
        }
    }
    // ---- sparse taps
    float ms_lo = L.owner ? m_lo : 1.0e30f, ms_hi = L.owner ? m_hi : 1.0e30f;   // what this lane subtracts
    // Folds G taps whose scores x0[i] (row g) and x1[i] (row g+8) are known into the running softmax.
    auto fold = [&](auto GC, const float (&x0)[decltype(GC)::value], const float (&x1)[decltype(GC)::value],
                    const RowFrag<D> (&vf0)[decltype(GC)::value], const RowFrag<D> (&vf1)[decltype(GC)::value]) {
        constexpr int G = decltype(GC)::value;
        float xm0 = x0[0], xm1 = x1[0];
#pragma unroll
        for (int i = 1; i < G; ++i) { xm0 = fmaxf(xm0, x0[i]); xm1 = fmaxf(xm1, x1[i]); }
        if (__any_sync(0xffffffffu, xm0 > ms_lo + kSlack || xm1 > ms_hi + kSlack)) {
            const float mn_lo = fmaxf(m_lo, __shfl_sync(0xffffffffu, xm0, L.owner_lane));
            const float mn_hi = fmaxf(m_hi, __shfl_sync(0xffffffffu, xm1, L.owner_lane));
            const float al_lo = ex2(m_lo - mn_lo), al_hi = ex2(m_hi - mn_hi);
            m_lo = mn_lo; m_hi = mn_hi;
            ms_lo = L.owner ? m_lo : 1.0e30f; ms_hi = L.owner ? m_hi : 1.0e30f;
            l_lo *= al_lo; l_hi *= al_hi;
#pragma unroll
            for (int j = 0; j < D / 8; ++j) { O[j][0] *= al_lo; O[j][1] *= al_lo; O[j][2] *= al_hi; O[j][3] *= al_hi; }
        }
#pragma unroll
        for (int i = 0; i < G; ++i) {
            const float p0 = ex2(x0[i] - ms_lo), p1 = ex2(x1[i] - ms_hi);   // exactly 0 on lanes that own no diagonal entry
            l_lo += p0; l_hi += p1;
            // P is diagonal: row g only needs its own value row, which this thread holds for the
            // same elements d as its accumulators
            diag_fma<D>(O, __shfl_sync(0xffffffffu, p0, L.owner_lane), __shfl_sync(0xffffffffu, p1, L.owner_lane),
                        vf0[i], vf1[i]);
        }
    };
    // G consecutive taps whose 16 key rows all exist: no predicates, loads of all G taps in flight together
    auto full_taps = [&](auto GC, int si) {
        constexpr int G = decltype(GC)::value;
        RowFrag<D> kf0[G], kf1[G], vf0[G], vf1[G];
        float pbv[G];
#pragma unroll
        for (int i = 0; i < G; ++i) {
            const int2 tp = make_int2(t.sparse[si + i], tap_s[si + i].y);
            pbv[i] = __int_as_float(tp.y);
            kr.template load2<AL>(kf0[i], kf1[i], -tp.x);
            vr.template load2<AL>(vf0[i], vf1[i], -tp.x);
        }
        float x0[G], x1[G];
#pragma unroll
        for (int i = 0; i < G; ++i) {
            float s0[4], s1[4];
            mma_rows_z(s0, qa, qb, kf0[i]);
            mma_rows_z(s1, qa, qb, kf1[i]);
            const float d0 = (g & 1) ? s0[1] : s0[0], d1 = (g & 1) ? s1[3] : s1[2];
            if constexpr (SE) {
                x0[i] = (d0 + qs0[si + i]) * c2;
                x1[i] = (d1 + qs1[si + i]) * c2;
            } else {
                x0[i] = fmaf(d0, c2, pbv[i]);
                x1[i] = fmaf(d1, c2, pbv[i]);
            }
        }
        fold(GC, x0, x1, vf0, vf1);
    };
    // A tile that reaches past row N-1 may pair its missing rows with key rows that do not exist
    // either (past the end of the sequence, for the last (b,h) past the end of the tensor).  Their
    // scores land in lanes that own no diagonal entry and are meant to contribute exp(x - 1e30) = 0;
    // a NaN or Inf bit pattern there would make that NaN, so boundary tiles take the predicated path,
    // which reads zeros for those rows.
    // Only interior tiles load taps unpredicated (boundary tiles are the first WB rows, which the
    // usual tap sets do not reach from, and the last partial tile).
    int si = 0;
    if constexpr (INTERIOR)
        for (; si + kTapGroup <= ns && g0 >= t.sparse[si + kTapGroup - 1]; si += kTapGroup)
            full_taps(std::integral_constant<int, kTapGroup>(), si);
#pragma unroll 1
    for (; si < ns; ++si) {
        const int delta = t.sparse[si];
        if (g0 + 15 < delta) break;                       // taps ascend: no row of the tile reaches back that far
        if (INTERIOR && g0 >= delta) {
            full_taps(std::integral_constant<int, 1>(), si);
        } else {                                          // some key rows lie outside the sequence
            const float pbv = __int_as_float(tap_s[si].y);
            const int kr0 = row_lo - delta, kr1 = row_hi - delta;
            const bool v0 = kr0 >= 0 && kr0 < N, v1 = kr1 >= 0 && kr1 < N;
            RowFrag<D> kf0, kf1, vf0[1], vf1[1];
            kr.template load2<AL>(kf0, kf1, -delta, v0, v1);
            vr.template load2<AL>(vf0[0], vf1[0], -delta, v0, v1);
            float s0[4], s1[4];
            mma_rows_z(s0, qa, qb, kf0);
            mma_rows_z(s1, qa, qb, kf1);
            const float d0 = (g & 1) ? s0[1] : s0[0], d1 = (g & 1) ? s1[3] : s1[2];
            const float y0 = SE ? (d0 + qs0[si]) * c2 : fmaf(d0, c2, pbv);
            const float y1 = SE ? (d1 + qs1[si]) * c2 : fmaf(d1, c2, pbv);
            const float x0[1] = {v0 ? y0 : kNeg};
            const float x1[1] = {v1 ? y1 : kNeg};
            fold(std::integral_constant<int, 1>(), x0, x1, vf0, vf1);
        }
    }
    l_lo = quad_sum(l_lo); l_hi = quad_sum(l_hi);
    const float gain = a.head_gain ? a.head_gain[h] : 1.f;
    __nv_bfloat16* op = static_cast<__nv_bfloat16*>(a.out) + obase;
    const float sc_lo = l_lo > 0.f ? __fdividef(gain, l_lo) : 0.f, sc_hi = l_hi > 0.f ? __fdividef(gain, l_hi) : 0.f;
    if (ST && a.gate) {
        const __nv_bfloat16* gp = static_cast<const __nv_bfloat16*>(a.gate) + (size_t)(bh / a.H) * a.gate_sb + (size_t)h * a.gate_sh;
        store_acc_rows_gated<D, AL>(O, op + (size_t)row_lo * OS, op + (size_t)row_hi * OS, gp + (size_t)row_lo * a.gate_sn,
                                    gp + (size_t)row_hi * a.gate_sn, ok_lo, ok_hi, sc_lo, sc_hi, tig);
    } else {
        store_acc_rows<D, AL>(O, op + (size_t)row_lo * OS, op + (size_t)row_hi * OS, ok_lo, ok_hi, sc_lo, sc_hi, tig);
    }
    if (tig == 0) {
        if (ok_lo) a.lse[(size_t)bh * N + row_lo] = l_lo > 0.f ? (m_lo + __log2f(l_lo)) * kLn2 : -INFINITY;
        if (ok_hi) a.lse[(size_t)bh * N + row_hi] = l_hi > 0.f ? (m_hi + __log2f(l_hi)) * kLn2 : -INFINITY;
    }
}

// Tuning per head dimension (measured on B200): warps per CTA, sparse taps folded together,
// resident CTAs per SM the register budget is set for.
template <int D> struct FwdTune {
    // Since a tap's address is one uniform product (Rows), registers allow more CTAs: D = 32 two taps, 7 CTAs (72 registers) 60.4 us at 32x8x2048,
    // 6 CTAs 64.1, 5 CTAs 66.8 (65.5 before); D = 64 79.7 us at 16x12x2048 (one tap 87.8, 5 CTAs 86.2; 92.4 before).
    // Swept on contiguous tensors only.  The strided and 16-byte instantiations take the same constants, although their 64-bit lane parts (Rows) need more
    // registers; bytes spilled (stores / loads), contiguous, strided, 16-byte: D = 32 32/32, 60/64, -; D = 64 0/0, 16/16, 48/48; with scale_embed D = 32
    // 0/0, 20/28, -; D = 64 12/20, 8/8, 24/28.  Packed forward with gate 32x8x2048x32 107 us.
    static constexpr int warps = 4, group = D > 96 ? 1 : 2, ctas = D == 32 ? 7 : (D <= 64 ? 4 : (D <= 96 ? 3 : 2));
    // With scale_embed a CTA first lays out the table, about a quarter of a tile's time, so a warp does up to three tiles with it.
    // The count is the one for which (waves of CTAs) x (tiles + 1/4) is least: one where the grid is a single wave (2x8x777x32 11.6 us,
    // 12.5 with two), two or three where that saves a wave or its table (4x8x2048x32 19.5 -> 18.7, 32x8x2048x32 101.4 -> 97.3,
    // 8x12x2048x64 73.9 -> 69.1; a fixed two would take 8x8x2048x32 from 30.0 to 33.1, three gives 28.9).
    static int tiles_se(int N, int BH) {
        int best = 1;
        long long least = 0;
        for (int t = 1; t <= 3; ++t) {
            const long long n = (long long)((N + 16 * warps * t - 1) / (16 * warps * t)) * BH, cost = (n + 148 * ctas_se - 1) / (148 * ctas_se) * (4 * t + 1);
            if (t == 1 || cost < least) { least = cost; best = t; }
        }
        return best;
    }
    static constexpr int group_se = 2, ctas_se = D == 32 ? 5 : 4;
};

// ST: addressing (kContiguous ...); with strides and a gate tensor the epilogue multiplies by sigmoid(gate).
template <int D, int WB, bool SE, int ST>
__global__ void __launch_bounds__(FwdTune<D>::warps * 32, SE ? FwdTune<D>::ctas_se : FwdTune<D>::ctas)
fwd_mma_kernel(const FwdArgs a, const Taps t, const int tiles_se) {
    stream_wait();
    constexpr int W = FwdTune<D>::warps, G = SE ? FwdTune<D>::group_se : FwdTune<D>::group;
    extern __shared__ __align__(16) float se_smem[];      // scale_embed: the table, then a tile per warp
    __shared__ __align__(16) float start_s[SE ? 4 : StartTable<WB>::kSize];
    __shared__ int2 tap_s[DSQG_MAX_TAPS];
    const Lane L;
    const int bh = blockIdx.y, h = bh % a.H, N = a.N;
    SeRows se = {};
    if constexpr (SE) {
        se = fill_se_rows<D, WB, W * 32>(se_smem, a.scale_embed, a.pos_bias, t, a.H, h, a.scale);
    } else {
        StartTable<WB>::template fill<false, W * 32>(start_s, a.pos_bias, a.H, h, t.d_lo, t.d_lo + t.n_dense - 1, a.scale);
    }
    for (int si = threadIdx.x; si < t.n_sparse; si += W * 32)
        tap_s[si] = make_int2(t.sparse[si], __float_as_int(a.pos_bias[(t.n_dense + si) * a.H + h] * kLog2e));
    __syncthreads();
    const float* start = StartTable<WB>::lane(start_s, L);
    float* se_tile = SE ? se_smem + se_rows_bytes<WB>(t.n_sparse, D) / 4 + L.warp * se_tile_floats<WB>(t.n_sparse) : se_smem;
    const int tiles = SE ? tiles_se : 1;
#pragma unroll 1
    for (int i = 0; i < tiles; ++i) {
        const int g0 = (blockIdx.x * tiles + i) * (16 * W) + L.warp * 16;
        if (g0 >= N) return;
        if (g0 >= WB && g0 + 16 <= N) fwd_tile<D, WB, true, G, SE, ST>(a, start, tap_s, t, t.n_sparse, bh, h, g0, L, se, se_tile);
        else fwd_tile<D, WB, false, G, SE, ST>(a, start, tap_s, t, t.n_sparse, bh, h, g0, L, se, se_tile);
        if (SE) __syncwarp();
    }
}

// Tuning per head dimension (measured on B200): sparse taps whose loads are issued together and
// resident CTAs per SM the register budget is set for (spills against warps in flight).
template <int D> struct BwdTune {
    // 8x8x2048 unless said otherwise, us: D = 32 at 32x8x2048 89.7 (6 CTAs 90.6, one tap and 6 CTAs 91.0, 4 CTAs 96.7), D = 64 at 16x12x2048
    // 114.9 (two taps 119.7), D = 80 59.8 (one tap 60.3), D = 96 66.0 (two taps 69.6, 2 CTAs 71.7-78.0), D = 128 84.5 (one tap 89.9).
    // All figures here are of contiguous tensors; the other instantiations take the same constants unswept (see FwdTune).  Bytes spilled (stores / loads),
    // contiguous, strided, 16-byte: dQ D = 32 48/52, 28/48, - (kept 48/52); D = 64 60/60, 100/124, 96/128; D = 96 12/12, 60/68, 68/76; with scale_embed
    // D = 64 28/40, 160/176, 104/124; dK/dV D = 64 16/16, 48/48, 20/20.  Packed backward with gate, us: 32x8x2048x32 191, 16x12x2048x64 297, 8x8x2048x128 248.5.
    static constexpr int dq_group = D == 64 || D == 96 ? 1 : 2, dq_ctas = D == 32 ? 5 : (D <= 64 ? 4 : (D <= 96 ? 3 : 2));
    // scale_embed: 32x8x2048x32 154.9 (5 CTAs 155.1, one tap 158-164), 16x12x2048x64 202.6 (one tap 208.6, 3 CTAs 205-212)
    static constexpr int dq_group_se = 2, dq_ctas_se = 4;
    // D = 32 at 32x8x2048 94.2 (4 CTAs 98.1, 6 CTAs 110-115), D = 64 at 16x12x2048 132.4 (two taps 134.9), D = 48 44.3, D = 80 69.0 (one tap 73.8,
    // 3 CTAs 82), D = 96 78.8 (one tap 82.1), D = 128 116.0 (two taps 125.2; two 16 x 128 accumulators and four row fragments do not fit 255
    // registers: 900 bytes spilled and 896 read back a thread, strided 1,144 / 1,152)
    static constexpr int dkdv_group = D == 64 ? 3 : (D > 96 ? 1 : 2), dkdv_ctas = D == 32 ? 5 : (D <= 64 ? 3 : 2);
    // scale_embed: 32x8x2048x32 129.1 (one tap 128.9, 4 CTAs 133.3), 16x12x2048x64 185.0 (two taps 187.1, 4 CTAs 238)
    static constexpr int dkdv_group_se = D == 32 ? 2 : 1, dkdv_ctas_se = D == 32 ? 5 : 3;
};
// Where a warp of the plain dQ kernel puts its ds values for dpos_bias.  Element (g + 8 half, 8 nt + 2 tig + c) of a
// tile belongs to offset g - 2 tig - c + 8 k with k = WB / 8 + half - nt, so elements of neighbouring n-tiles share
// (lane, c, k) and are added in registers first: 2 (WB/8 + 3) stores per lane instead of 4 (WB/8 + 2), to [c][k + 1][lane];
// then one lane per offset adds the eight entries of its offset in a fixed order.  The pitch of 33 makes these reads
// (stride 4 in g, 1 in k) conflict-free.  Sparse taps: one value per row pair to [g][tap].
template <int WB> struct DsStage {
    static constexpr int kK = WB / 8 + 3, kDense = 2 * kK * 33;
    static __host__ __device__ int sparse_pitch(int ns) { return ns | 1; }
    static __host__ __device__ int floats(int ns, int J) { return kDense + 8 * sparse_pitch(ns) + J; }    // per warp, with its J sums
    static __device__ __forceinline__ void put(float* w, int lane, int k1, float a, float b) {
        w[k1 * 33 + lane] = a;
        w[(kK + k1) * 33 + lane] = b;
    }
    static __device__ __forceinline__ void sum(float* w, const Taps& t, int lane) {
        const float* sp = w + kDense;
        const int pitch = sparse_pitch(t.n_sparse);
        float* out = w + kDense + 8 * pitch;
        __syncwarp();
        for (int j = lane; j < t.n_dense; j += 32) {
            float s[2] = {0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int e = t.d_lo + j + 2 * i + c;              // = g + 8 k
                    s[c] += w[(c * kK + (e >> 3) + 1) * 33 + 4 * (e & 7) + i];
                }
            out[j] = s[0] + s[1];
        }
        for (int j = lane; j < t.n_sparse; j += 32) {
            float s = 0.f;
#pragma unroll
            for (int g = 0; g < 8; ++g) s += sp[g * pitch + j];
            out[t.n_dense + j] = s;
        }
    }
};

// Extras of the dQ kernel with scale_embed.  A warp's tile of start values (build_se_tile) becomes its tile of ds values: every
// element is read and then overwritten by the lane that owns it, and the sparse taps follow the dense ones at column
// WB + 17, so that columns 16 .. 16 (steps + 1) are dS in the order of the table rows.  The products dS.SE take their operand from there; its
// bf16 fragments are also stored row by row (ds16), from where ldmatrix.trans hands them to the products dS^T.Q of the whole CTA
// (four words of the fp32 tile per fragment register instead: dQ stage at 32x8x2048x32 172 us, now 162 us; 16x12x2048x64 231 and 216 us).
template <int WB> struct SeBwd {
    SeRows rows;
    const uint2* seb;            // table as B fragments of dS.SE (global memory, written by se_prep_kernel)
    unsigned char* q_s;          // the CTA's 64 query rows as bf16 in shared memory, row pitch 2D+16 bytes (conflict-free ldmatrix)
    float* tile; float* sparse;  // this warp's
    unsigned char* ds16;         // this warp's 16 rows of dS as bf16, row pitch pitch16 bytes (an odd multiple of 16: conflict-free)
    int pitch, sp, pitch16;
    static constexpr int kSparse = WB + 17;                                                              // column of the first sparse tap
    static __host__ __device__ int steps(int ns) { return (WB + 1 + ns + 15) / 16; }                      // 16-column steps of dS
    static __host__ __device__ int pitch_for(int ns) {                                                    // 9 mod 32
        const int need = steps(ns) * 16 + 16 > WB + 32 ? steps(ns) * 16 + 16 : WB + 32;
        return (need - 9 + 31) / 32 * 32 + 9;
    }
    // floats per warp; the odd multiple of 8 puts the tiles two warps apart 16 banks apart (column sums)
    static __host__ __device__ int floats(int ns) { return 16 * (pitch_for(ns) + SeGeo<WB>::sparse_pitch(ns)) + 8; }
    static __host__ __device__ int pitch16_for(int ns) { return 32 * steps(ns) + 16; }
    // tap of column 16 + p of dS, -1: none
    static __device__ __forceinline__ int tap(const Taps& t, int p) {
        const int j = p <= WB ? WB - p - t.d_lo : t.n_dense + p - WB - 1;
        return p <= WB ? (j >= 0 && j < t.n_dense ? j : -1) : (j < t.J ? j : -1);
    }
};

template <int D, int WB, bool INTERIOR, int G, bool SE, int ST>
__device__ __forceinline__ float dq_tile(const BwdArgs& a, const float* start, const int2* tap_s,
                                         float* stage_w, const Taps& t, int ns, int bh, int h, int g0, const Lane& L, const SeBwd<WB>& sb) {
    constexpr int NT = (WB + 16) / 8;
    using Stage = DsStage<WB>;
    const int N = a.N, g = L.g, tig = L.tig;
    const int row_lo = g0 + g, row_hi = row_lo + 8;
    const bool ok_lo = INTERIOR || row_lo < N, ok_hi = INTERIOR || row_hi < N;
    constexpr bool AL = ST != kStridedAny, CI = ST == kContiguous || ST == kKept;          // CI: what is read is contiguous
    const ptrdiff_t GS = ST ? (ptrdiff_t)a.in_sn : D, RS = CI ? D : GS, OS = CI ? D : (ptrdiff_t)a.out_sn;   // row strides of dq, q/k/v, out/dout
    const size_t cbase = (size_t)bh * N * D, gbase = ST ? (size_t)(bh / a.H) * a.in_sb + (size_t)h * a.in_sh : cbase, base = CI ? cbase : gbase;
    const size_t obase = CI ? cbase : (size_t)(bh / a.H) * a.out_sb + (size_t)h * a.out_sh;
    const Rows<D, CI> qr(a.q, base, g0, RS, L), kr(a.k, base, g0, RS, L), vr(a.v, base, g0, RS, L);
    const Rows<D, CI> orow(a.out, obase, g0, OS, L), dr(a.dout, obase, g0, OS, L);
    const float c2 = a.scale * kLog2e;
    const float gain = a.head_gain ? a.head_gain[h] : 1.f;
    const int kb0 = g0 - WB;
    float dgrow = 0.f;
    f32x2 dgrow2 = 0ull;

    RowFrag<D> qa, qb, da, db;
    float delta_lo, delta_hi;
    bool have_dout = ST != kKept;
    if constexpr (ST != kContiguous) have_dout = have_dout && !a.gate;
    if constexpr (ST != kContiguous) if (!have_dout) {       // the gate's backward for these rows first
        auto rows = [&](const void* p, const dsqg_strides& st) {
            return Rows<D, false>(p, (size_t)(bh / a.H) * st.batch + (size_t)h * st.head, g0, (ptrdiff_t)st.row, L);
        };
        RowFrag<D> ya, yb, ga, gb;
        rows(a.dy, a.y_st).template load2<AL>(da, db, 0, ok_lo, ok_hi);
        rows(a.y, a.y_st).template load2<AL>(ya, yb, 0, ok_lo, ok_hi);
        rows(a.gate, a.gate_st).template load2<AL>(ga, gb, 0, ok_lo, ok_hi);
        delta_lo = row_dot(da, ya); delta_hi = row_dot(db, yb);
        gate_row(da, ya, ga); gate_row(db, yb, gb);
        const Rows<D, false> dg = rows(a.dgate, a.dgate_st);
        if (ok_lo) {
            store_row_at<D, AL>(ya.r, const_cast<__nv_bfloat16*>(dg.at(0)));
            store_row_at<D, AL>(da.r, const_cast<__nv_bfloat16*>(dr.at(0)));
        }
        if (ok_hi) {
            store_row_at<D, AL>(yb.r, const_cast<__nv_bfloat16*>(dg.at(8)));
            store_row_at<D, AL>(db.r, const_cast<__nv_bfloat16*>(dr.at(8)));
        }
    }
    qr.template load2<AL>(qa, qb, 0, ok_lo, ok_hi);
    if (have_dout) dr.template load2<AL>(da, db, 0, ok_lo, ok_hi);
    if constexpr (SE) {
        // the sparse part also goes to global memory for the dK/dV kernel (a row of ns8 floats per query)
        const int ns8 = (ns + 7) / 8 * 8;
        float* rows = a.qs_rows + ((size_t)bh * N + row_lo) * ns8;
        build_se_tile<D, WB, true>(sb.rows, ns, qa, qb, g, tig, sb.tile, sb.pitch, sb.sparse, sb.sp, ok_lo ? rows : nullptr,
                                   ok_hi ? rows + 8 * ns8 : nullptr);
        // and the query rows to shared memory for the CTA's dscale_embed partial
        unsigned char* qrow = sb.q_s + (size_t)(L.warp * 16 + g) * (2 * D + 16) + 2 * kLane<D> * tig;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
            const int o = kLane<D> == 16 ? 128 * (c >> 1) + 16 * (c & 1) : 64 * c;
            *reinterpret_cast<uint4*>(qrow + o) = make_uint4(qa.r[4 * c], qa.r[4 * c + 1], qa.r[4 * c + 2], qa.r[4 * c + 3]);
            *reinterpret_cast<uint4*>(qrow + 8 * (2 * D + 16) + o) = make_uint4(qb.r[4 * c], qb.r[4 * c + 1], qb.r[4 * c + 2], qb.r[4 * c + 3]);
        }
    }
    if (ST && ST != kKept && have_dout && a.delta_pre) {       // sum_d dout*out was handed in by a caller of the strided entries
        delta_lo = ok_lo ? a.delta_pre[(size_t)bh * N + row_lo] : 0.f;
        delta_hi = ok_hi ? a.delta_pre[(size_t)bh * N + row_hi] : 0.f;
    } else if (have_dout) {
        RowFrag<D> oa, ob;
        orow.template load2<AL>(oa, ob, 0, ok_lo, ok_hi);
        delta_lo = quad_sum(frag_dot(da, oa));
        delta_hi = quad_sum(frag_dot(db, ob));
    }
    float l2_lo = 0.f, l2_hi = 0.f;
    if (ok_lo) { const float x = a.lse[(size_t)bh * N + row_lo]; l2_lo = x == -INFINITY ? 0.f : x * kLog2e; }
    if (ok_hi) { const float x = a.lse[(size_t)bh * N + row_hi]; l2_hi = x == -INFINITY ? 0.f : x * kLog2e; }
    if (tig == 0) {
        float2* rs = reinterpret_cast<float2*>(a.delta) + (size_t)bh * N;
        if (ok_lo) rs[row_lo] = make_float2(l2_lo, delta_lo);
        if (ok_hi) rs[row_hi] = make_float2(l2_hi, delta_hi);
    }
    float dQ[D / 8][4];
    float carry[2] = {0.f, 0.f};                                   // plain kernel: row g's ds of the n-tile before
    float* se_lane = SE ? sb.tile + g * (sb.pitch - 1) + 16 + 2 * tig : nullptr;

    // ---- dense window
    const __nv_bfloat16 *k_band = kr.at(-WB), *v_band = vr.at(-WB);
#pragma unroll
    for (int c = 0; c < NT / 2; ++c) {
        RowFrag<D> kf[2];
        float ds[2][4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int nt = 2 * c + hf;
            float s[4], dp[4];
            if constexpr (SE) {
                se_start<WB>(s, se_lane, sb.pitch, nt, g, tig);
            } else {
                StartTable<WB>::get(s, start, nt);
            }
            RowFrag<D> vf;
            const __nv_bfloat16* kp = CI ? k_band + 8 * nt * D : kr.at(8 * nt - WB);
            const __nv_bfloat16* vp = CI ? v_band + 8 * nt * D : vr.at(8 * nt - WB);
            if (INTERIOR) {
                load_row_at<D, AL>(kf[hf], kp);
                load_row_at<D, AL>(vf, vp);
            } else {
                const int r = kb0 + 8 * nt + g;
                const bool valid = r >= 0 && r < N;
                load_piece<D, AL>(kf[hf], kp, valid);
                load_piece<D, AL>(vf, vp, valid);
            }
            mma_rows(s, qa, qb, kf[hf]);
            mma_rows_z(dp, da, db, vf);
            if (!INTERIOR && kb0 < 0) {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (kb0 + 8 * nt + 2 * tig + (r & 1) < 0) s[r] = kNeg;
            }
#pragma unroll
            for (int r = 0; r < 4; r += 2) {
                const float l = r ? l2_hi : l2_lo, d = r ? delta_hi : delta_lo;
                float p0, p1;
                unpair(fma2(pair(s[r], s[r + 1]), pair(c2, c2), pair(-l, -l)), p0, p1);
                const f32x2 pp = pair(ex2(p0), ex2(p1)), dpp = pair(dp[r], dp[r + 1]);
                dgrow2 = fma2(pp, dpp, dgrow2);
                unpair(mul2(pp, fma2(pair(gain, gain), dpp, pair(-d, -d))), ds[hf][r], ds[hf][r + 1]);
            }
            if constexpr (SE) {
                *reinterpret_cast<float2*>(se_lane + 8 * nt) = make_float2(ds[hf][0], ds[hf][1]);
                if (nt > 0) *reinterpret_cast<float2*>(se_lane + 8 * (sb.pitch - 1) + 8 * nt) = make_float2(ds[hf][2], ds[hf][3]);
            }
            if constexpr (!SE) {
                Stage::put(stage_w, L.lane, WB / 8 + 2 - nt, nt ? carry[0] + ds[hf][2] : ds[hf][2], nt ? carry[1] + ds[hf][3] : ds[hf][3]);
                carry[0] = ds[hf][0]; carry[1] = ds[hf][1];
            }
        }
        RowFrag<D> kt0, kt1;
        transpose_frag(kt0, kf[0]); transpose_frag(kt1, kf[1]);
        const uint32_t a0 = pack_bf16x2(ds[0][0], ds[0][1]), a1 = pack_bf16x2(ds[0][2], ds[0][3]);
        const uint32_t a2 = pack_bf16x2(ds[1][0], ds[1][1]), a3 = pack_bf16x2(ds[1][2], ds[1][3]);
        if (c == 0) {
#pragma unroll
            for (int j = 0; j < D / 8; ++j) mma16816_z(dQ[j], a0, a1, a2, a3, kt0.r[j], kt1.r[j]);
        } else {
            mma_cols<D>(dQ, a0, a1, a2, a3, kt0, kt1);
        }
    }
    // ---- sparse taps
    const float ls_lo = L.owner ? l2_lo : 1.0e30f, ls_hi = L.owner ? l2_hi : 1.0e30f;   // p == 0 on lanes without a diagonal entry
    if constexpr (!SE) Stage::put(stage_w, L.lane, 0, carry[0], carry[1]);
    // one value per sparse tap: row pairs' sums in the plain kernel, rows g and g + 8 with scale_embed
    float* stage_sp = SE ? sb.tile + g * sb.pitch + SeBwd<WB>::kSparse : stage_w + Stage::kDense + g * Stage::sparse_pitch(ns);
    const int stage_hi = SE ? 8 * sb.pitch : 0;
    const float* qs0 = SE ? sb.sparse + g * sb.sp : nullptr;
    const float* qs1 = qs0 + 8 * sb.sp;
    if constexpr (SE) {
        __syncwarp();                                     // the dense columns' owners have written what lies under the sparse ones
        const int first = SeBwd<WB>::kSparse + ns, pad = 16 * SeBwd<WB>::steps(ns) + 16 - first;
        for (int e = L.lane; e < 16 * pad; e += 32) sb.tile[(e & 15) * sb.pitch + first + (e >> 4)] = 0.f;
    }
    auto finish = [&](int si, float sd0, float sd1, float dp0, float dp1, float pbv, bool v0, bool v1,
                      const RowFrag<D>& kf0, const RowFrag<D>& kf1) {
        float p0, p1;
        if constexpr (SE) {
            p0 = v0 ? ex2((sd0 + qs0[si]) * c2 - ls_lo) : 0.f;
            p1 = v1 ? ex2((sd1 + qs1[si]) * c2 - ls_hi) : 0.f;
        } else {
            p0 = v0 ? ex2(fmaf(sd0, c2, pbv) - ls_lo) : 0.f;
            p1 = v1 ? ex2(fmaf(sd1, c2, pbv) - ls_hi) : 0.f;
        }
        dgrow = fmaf(p0, dp0, dgrow); dgrow = fmaf(p1, dp1, dgrow);
        const float x0 = p0 * fmaf(gain, dp0, -delta_lo), x1 = p1 * fmaf(gain, dp1, -delta_hi);
        if (L.owner) {
            if constexpr (SE) { stage_sp[si] = x0; stage_sp[stage_hi + si] = x1; } else stage_sp[si] = x0 + x1;
        }
        diag_fma<D>(dQ, __shfl_sync(0xffffffffu, x0, L.owner_lane), __shfl_sync(0xffffffffu, x1, L.owner_lane), kf0, kf1);
    };
    auto full_taps = [&](auto GC, int si) {
        constexpr int GG = decltype(GC)::value;
        RowFrag<D> kf0[GG], kf1[GG], vf0[GG], vf1[GG];
        float pbv[GG];
#pragma unroll
        for (int i = 0; i < GG; ++i) {
            const int2 tp = make_int2(t.sparse[si + i], tap_s[si + i].y);
            pbv[i] = __int_as_float(tp.y);
            kr.template load2<AL>(kf0[i], kf1[i], -tp.x);
            vr.template load2<AL>(vf0[i], vf1[i], -tp.x);
        }
#pragma unroll
        for (int i = 0; i < GG; ++i) {
            float s0[4], s1[4], e0[4], e1[4];
            mma_rows_z(s0, qa, qb, kf0[i]); mma_rows_z(s1, qa, qb, kf1[i]);
            mma_rows_z(e0, da, db, vf0[i]); mma_rows_z(e1, da, db, vf1[i]);
            finish(si + i, (g & 1) ? s0[1] : s0[0], (g & 1) ? s1[3] : s1[2], (g & 1) ? e0[1] : e0[0],
                   (g & 1) ? e1[3] : e1[2], pbv[i], true, true, kf0[i], kf1[i]);
        }
    };
    // as in the forward: only interior tiles load taps unpredicated, so no key row past the end is read
    int si = 0;
    if constexpr (INTERIOR)
        for (; si + G <= ns && g0 >= t.sparse[si + G - 1]; si += G) full_taps(std::integral_constant<int, G>(), si);
#pragma unroll 1
    for (; si < ns; ++si) {
        const int delta = t.sparse[si];
        if (g0 + 15 < delta) break;
        if (INTERIOR && g0 >= delta) {
            full_taps(std::integral_constant<int, 1>(), si);
        } else {
            const float pbv = __int_as_float(tap_s[si].y);
            const bool v0 = row_lo >= delta && row_lo - delta < N, v1 = row_hi >= delta && row_hi - delta < N;
            RowFrag<D> kf0, kf1, vf0, vf1;
            kr.template load2<AL>(kf0, kf1, -delta, v0, v1);
            vr.template load2<AL>(vf0, vf1, -delta, v0, v1);
            float s0[4], s1[4], e0[4], e1[4];
            mma_rows_z(s0, qa, qb, kf0); mma_rows_z(s1, qa, qb, kf1);
            mma_rows_z(e0, da, db, vf0); mma_rows_z(e1, da, db, vf1);
            finish(si, (g & 1) ? s0[1] : s0[0], (g & 1) ? s1[3] : s1[2], (g & 1) ? e0[1] : e0[0],
                   (g & 1) ? e1[3] : e1[2], pbv, v0, v1, kf0, kf1);
        }
    }
    if (L.owner)                                          // taps no row of the tile reaches: zero entries
        for (; si < ns; ++si) {
            stage_sp[si] = 0.f;
            if constexpr (SE) stage_sp[stage_hi + si] = 0.f;
        }
    if constexpr (SE) {
        // dQ += dS.scale_embed: the warp's ds values are complete in its tile
        __syncwarp();
#pragma unroll 1
        for (int kk = 0; kk < SeBwd<WB>::steps(ns); ++kk) {
            const float* lo = sb.tile + g * sb.pitch + 16 + 16 * kk + 2 * tig;
            const float* hi = lo + 8 * sb.pitch;
            const uint32_t a0 = pack_bf16x2(lo[0], lo[1]), a1 = pack_bf16x2(hi[0], hi[1]);
            const uint32_t a2 = pack_bf16x2(lo[8], lo[9]), a3 = pack_bf16x2(hi[8], hi[9]);
            unsigned char* d16 = sb.ds16 + g * sb.pitch16 + 32 * kk + 4 * tig;
            *reinterpret_cast<uint32_t*>(d16) = a0; *reinterpret_cast<uint32_t*>(d16 + 16) = a2;
            *reinterpret_cast<uint32_t*>(d16 + 8 * sb.pitch16) = a1; *reinterpret_cast<uint32_t*>(d16 + 8 * sb.pitch16 + 16) = a3;
#pragma unroll
            for (int jn = 0; jn < D / 8; ++jn) {
                const uint2 b = __ldg(sb.seb + (kk * (D / 8) + jn) * 32 + L.lane);
                mma16816(dQ[jn], a0, a1, a2, a3, b.x, b.y);
            }
        }
    }
    __nv_bfloat16* dqp = static_cast<__nv_bfloat16*>(a.dq) + gbase;
    store_acc_rows<D, AL>(dQ, dqp + (size_t)row_lo * GS, dqp + (size_t)row_hi * GS, ok_lo, ok_hi, a.scale, a.scale, tig);
    float dg0, dg1;
    unpair(dgrow2, dg0, dg1);
    return dgrow + (dg0 + dg1);
}

// One block, before the dQ kernel with scale_embed.  Writes, back to back: the table (SeRows) as bf16 halves [2][R][D]; its B fragments for
// dQ += dS.scale_embed, [steps][D/8][32] x uint2, in the element order of the dQ accumulators (row fragment register jn of lane
// tig = g>>1, element g&1); pos_bias / scale or the mask value for every head, [H][R].
struct SePre {
    const __nv_bfloat16* hi; const __nv_bfloat16* lo; const uint2* seb; const float* pb;
};
template <int WB>
__host__ __device__ inline SePre se_pre_layout(const void* base, int ns, int D) {
    const int R = SeGeo<WB>::rows(ns);
    SePre p;
    p.hi = static_cast<const __nv_bfloat16*>(base);
    p.lo = p.hi + R * D;
    p.seb = reinterpret_cast<const uint2*>(p.lo + R * D);
    p.pb = reinterpret_cast<const float*>(p.seb + SeBwd<WB>::steps(ns) * (D / 8) * 32);
    return p;
}
template <int D, int WB>
__global__ void se_prep_kernel(const float* __restrict__ scale_embed, const float* __restrict__ pos_bias, float scale, const Taps t, int H, void* out) {
    stream_wait();
    const SePre P = se_pre_layout<WB>(out, t.n_sparse, D);
    const int R = SeGeo<WB>::rows(t.n_sparse);
    __nv_bfloat162* hi = reinterpret_cast<__nv_bfloat162*>(const_cast<__nv_bfloat16*>(P.hi));
    __nv_bfloat162* lo = reinterpret_cast<__nv_bfloat162*>(const_cast<__nv_bfloat16*>(P.lo));
    for (int e = threadIdx.x; e < R * D / 2; e += blockDim.x) {
        const int j = SeGeo<WB>::tap(t, 2 * e / D);
        float2 x = make_float2(0.f, 0.f);
        if (j >= 0) x = *reinterpret_cast<const float2*>(scale_embed + j * D + 2 * e % D);
        const __nv_bfloat162 h2 = __floats2bfloat162_rn(x.x, x.y);
        hi[e] = h2;
        lo[e] = __floats2bfloat162_rn(x.x - __low2float(h2), x.y - __high2float(h2));
    }
    uint2* seb = const_cast<uint2*>(P.seb);
    for (int e = threadIdx.x; e < SeBwd<WB>::steps(t.n_sparse) * (D / 8) * 32; e += blockDim.x) {
        const int ln = e & 31, jn = (e >> 5) % (D / 8), kk = (e >> 5) / (D / 8);
        const int gg = ln >> 2, tt = ln & 3;
        constexpr int kPer = kLane<D> / 2;                       // n-tiles per piece
        const int d = 4 * kLane<D> * (jn / kPer) + kLane<D> * (gg >> 1) + 2 * (jn % kPer) + (gg & 1);
        auto sev = [&](int p) { const int j = SeBwd<WB>::tap(t, p); return j >= 0 ? scale_embed[j * D + d] : 0.f; };
        const int p0 = 16 * kk + 2 * tt;
        seb[e] = make_uint2(pack_bf16x2(sev(p0), sev(p0 + 1)), pack_bf16x2(sev(p0 + 8), sev(p0 + 9)));
    }
    float* pb = const_cast<float*>(P.pb);
    const float inv_scale = 1.f / scale;
    for (int e = threadIdx.x; e < H * R; e += blockDim.x) {
        const int h = e / R, j = SeGeo<WB>::tap(t, e - h * R);
        pb[e] = j >= 0 ? pos_bias[j * H + h] * inv_scale : kNeg;
    }
}

// [kWarps] dgain terms, then per warp a DsStage or, with scale_embed, a SeBwd tile; then the query rows and dS as bf16
template <int D, int WB>
inline size_t dq_smem_bytes(int J, int ns, bool se) {
    return sizeof(float) * kWarps * (size_t)(1 + (se ? SeBwd<WB>::floats(ns) : DsStage<WB>::floats(ns, J))) + (se ? (size_t)kRows * (2 * D + 16 + SeBwd<WB>::pitch16_for(ns)) : 0);
}

template <int D, int WB, int G, int CT, bool SE, int ST>
__global__ void __launch_bounds__(kWarps * 32, CT)
bwd_dq_mma_kernel(const BwdArgs a, const Taps t) {
    stream_wait();
    using Stage = DsStage<WB>;
    extern __shared__ __align__(16) float stage[];     // see dq_smem_bytes
    __shared__ __align__(16) float start_s[SE ? 4 : StartTable<WB>::kSize];
    __shared__ int2 tap_s[DSQG_MAX_TAPS];
    const Lane L;
    const int bh = blockIdx.y, h = bh % a.H, N = a.N, J = t.J;
    float* dg_s = stage;
    SeBwd<WB> sb = {};
    if constexpr (!SE) StartTable<WB>::template fill<false, kWarps * 32>(start_s, a.pos_bias, a.H, h, t.d_lo, t.d_lo + t.n_dense - 1, a.scale);
    for (int si = threadIdx.x; si < t.n_sparse; si += kWarps * 32)
        tap_s[si] = make_int2(t.sparse[si], __float_as_int(a.pos_bias[(t.n_dense + si) * a.H + h] * kLog2e));
    const int per_se = SE ? SeBwd<WB>::floats(t.n_sparse) : 0;
    if constexpr (SE) {
        const SePre P = se_pre_layout<WB>(a.se_pre, t.n_sparse, D);
        sb.rows = {P.hi, P.lo, P.pb + h * SeGeo<WB>::rows(t.n_sparse)};
        sb.seb = P.seb;
        sb.pitch = SeBwd<WB>::pitch_for(t.n_sparse); sb.sp = SeGeo<WB>::sparse_pitch(t.n_sparse);
        sb.tile = stage + kWarps + L.warp * per_se;
        sb.sparse = sb.tile + 16 * sb.pitch;
        sb.q_s = reinterpret_cast<unsigned char*>(stage + kWarps + kWarps * per_se);
        sb.pitch16 = SeBwd<WB>::pitch16_for(t.n_sparse);
        sb.ds16 = sb.q_s + kRows * (2 * D + 16) + L.warp * 16 * sb.pitch16;
    }
    __syncthreads();
    const int g0 = blockIdx.x * kRows + L.warp * 16;
    float* stage_w = stage + kWarps + L.warp * Stage::floats(t.n_sparse, J);                     // plain kernel
    float* sums = stage + kWarps + Stage::kDense + 8 * Stage::sparse_pitch(t.n_sparse);          // plain kernel: warp 0's J sums
    const float* start = StartTable<WB>::lane(start_s, L);
    float dgrow = 0.f;
    if (g0 >= N) {                                      // no rows: this warp's sums, or ds tile and query rows, are zero
        if constexpr (SE) {
            for (int e = L.lane; e < 16 * sb.pitch; e += 32) sb.tile[e] = 0.f;
        } else {
            for (int j = L.lane; j < J; j += 32) sums[L.warp * Stage::floats(t.n_sparse, J) + j] = 0.f;
        }
        if constexpr (SE)
            for (int e = L.lane; e < 16 * (2 * D + 16) / 16; e += 32)
                reinterpret_cast<uint4*>(sb.q_s + (size_t)L.warp * 16 * (2 * D + 16))[e] = make_uint4(0u, 0u, 0u, 0u);
        if constexpr (SE)
            for (int e = L.lane; e < sb.pitch16; e += 32) reinterpret_cast<uint4*>(sb.ds16)[e] = make_uint4(0u, 0u, 0u, 0u);
    } else if (g0 >= WB && g0 + 16 <= N) {
        dgrow = dq_tile<D, WB, true, G, SE, ST>(a, start, tap_s, stage_w, t, t.n_sparse, bh, h, g0, L, sb);
    } else {
        dgrow = dq_tile<D, WB, false, G, SE, ST>(a, start, tap_s, stage_w, t, t.n_sparse, bh, h, g0, L, sb);
    }
    if constexpr (!SE)
        if (g0 < N) Stage::sum(stage_w, t, L.lane);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dgrow += __shfl_xor_sync(0xffffffffu, dgrow, o);
    if (L.lane == 0) dg_s[L.warp] = dgrow;
    __syncthreads();
    const int tile = bh * a.tiles_per_bh + blockIdx.x;
    if constexpr (SE) {
        // CTA partial of dscale_embed = scale * dS^T . Q[64 x D]; warp w takes n-tiles w, w+4, ...
        constexpr int QP = 2 * D + 16;
        const uint32_t q_base = static_cast<uint32_t>(__cvta_generic_to_shared(sb.q_s));
        const uint32_t ds_base = q_base + kRows * QP + ((L.lane & 7) + (L.lane >> 4) * 8) * sb.pitch16 + ((L.lane >> 3) & 1) * 16;
#pragma unroll 1
        for (int jn = L.warp; jn < D / 8; jn += kWarps) {
#pragma unroll 1
            for (int mt = 0; mt < SeBwd<WB>::steps(t.n_sparse); ++mt) {
                float c[4];
#pragma unroll
                for (int kk = 0; kk < kRows / 16; ++kk) {
                    uint32_t a0, a1, a2, a3, b0, b1;
                    const uint32_t q_at = q_base + (16 * kk + (L.lane & 15)) * QP + 16 * jn, ds_at = ds_base + 16 * kk * sb.pitch16 + 32 * mt;
                    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(b0), "=r"(b1) : "r"(q_at));
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3) : "r"(ds_at));
                    if (kk == 0) mma16816_z(c, a0, a1, a2, a3, b0, b1); else mma16816(c, a0, a1, a2, a3, b0, b1);
                }
                // the tile's partial goes to global memory; dse_group_kernel adds the tiles of a group
                const int j0 = SeBwd<WB>::tap(t, 16 * mt + L.g), j1 = SeBwd<WB>::tap(t, 16 * mt + L.g + 8);
                float* dst = a.dse_tmp + (size_t)tile * J * D + 8 * jn + 2 * L.tig;
                if (j0 >= 0) *reinterpret_cast<float2*>(dst + j0 * D) = make_float2(c[0] * a.scale, c[1] * a.scale);
                if (j1 >= 0) *reinterpret_cast<float2*>(dst + j1 * D) = make_float2(c[2] * a.scale, c[3] * a.scale);
            }
        }
    }
    if constexpr (!SE) {
        static_assert(kWarps == 4, "four warps' sums");
        const int per = Stage::floats(t.n_sparse, J);
        for (int j = threadIdx.x; j < J; j += kWarps * 32)
            a.dpb_part[(size_t)tile * J + j] = (sums[j] + sums[per + j]) + (sums[2 * per + j] + sums[3 * per + j]);
    } else {
        // Column sums of the ds tiles: two threads per tap (two tiles each, fixed order); half 1's tiles lie 16 banks from half 0's
        static_assert(kWarps == 4, "two tiles per thread");
        for (int p0 = 0; p0 < 16 * SeBwd<WB>::steps(t.n_sparse); p0 += kWarps * 16) {
            const int p = p0 + (threadIdx.x >> 1), half = threadIdx.x & 1;
            const int j = p < 16 * SeBwd<WB>::steps(t.n_sparse) ? SeBwd<WB>::tap(t, p) : -1;
            float s = 0.f;
            if (j >= 0) {
                const float* u = stage + kWarps + 2 * half * per_se + 16 + p;
                float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
                for (int r = 0; r < 16; r += 2) {
                    s0 += u[r * sb.pitch]; s1 += u[(r + 1) * sb.pitch];
                    s2 += u[per_se + r * sb.pitch]; s3 += u[per_se + (r + 1) * sb.pitch];
                }
                s = (s0 + s1) + (s2 + s3);
            }
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            if (j >= 0 && half == 0) a.dpb_part[(size_t)tile * J + j] = s;
        }
    }
    if (threadIdx.x == 0) a.dg_part[tile] = (dg_s[0] + dg_s[1]) + (dg_s[2] + dg_s[3]);
}

// dscale_embed partials: one block per group of kSeGroup consecutive 64-row tiles of a sequence adds
// the tiles' partials (written by the dQ kernel) in tile order.
__global__ void __launch_bounds__(256)
dse_group_kernel(const float* __restrict__ tmp, float* __restrict__ part, int tiles_per_bh, int groups_bh, int JD) {
    stream_wait();
    const int bh = blockIdx.y, grp = blockIdx.x, first = grp * kSeGroup;
    const int members = tiles_per_bh - first < kSeGroup ? tiles_per_bh - first : kSeGroup;
    const float* src = tmp + ((size_t)bh * tiles_per_bh + first) * JD;
    float* out = part + ((size_t)bh * groups_bh + grp) * JD;
    for (int e = threadIdx.x; e < JD; e += 256) {
        float x[kSeGroup];
#pragma unroll
        for (int r = 0; r < kSeGroup; ++r) x[r] = r < members ? __ldg(src + (size_t)r * JD + e) : 0.f;
        float s = x[0];
#pragma unroll
        for (int r = 1; r < kSeGroup; ++r) s += x[r];
        out[e] = s;
    }
}

// ------------------------------------------------------------------------------ backward: dK, dV
// The warp owns 16 key rows; the roles of rows and columns are swapped: S^T = K.Q^T over the
// query rows [m0, m0+16+WB) for the dense window and the diagonal of the tile at m0+delta for
// every sparse tap.  Key rows are owned by exactly one warp: no atomics.  The per-query
// statistics {lse*log2(e), delta} of the CTA's dense query range sit in shared memory.
// With scale_embed the CTA forms q.scale_embed of its dense query range once more (build_se_tile, 16 rows per warp and step) instead of
// reading a per-row table of it from global memory; the score accumulators of the dense window start from that tile, and a
// sparse tap adds the entry of its query row, which the dQ kernel left in qs_rows.
template <int D, int WB, bool INTERIOR, int G, bool SE, int ST>
__device__ __forceinline__ void dkdv_tile(const BwdArgs& a, const float* start, const int2* tap_s, const float* stat_w,
                                          const Taps& t, int ns, int bh, int h, int m0, const Lane& L, const float* se_tile) {
    constexpr int NT = (WB + 16) / 8, kStat = kRows + WB;
    const int N = a.N, g = L.g, tig = L.tig;
    const int row_lo = m0 + g, row_hi = row_lo + 8;
    const bool ok_lo = INTERIOR || row_lo < N, ok_hi = INTERIOR || row_hi < N;
    constexpr bool AL = ST != kStridedAny, CI = ST == kContiguous || ST == kKept;          // CI: what is read is contiguous
    const ptrdiff_t GS = ST ? (ptrdiff_t)a.in_sn : D, RS = CI ? D : GS, OS = CI ? D : (ptrdiff_t)a.out_sn;   // row strides of dk/dv, q/k/v, dout
    const size_t cbase = (size_t)bh * N * D, gbase = ST ? (size_t)(bh / a.H) * a.in_sb + (size_t)h * a.in_sh : cbase, base = CI ? cbase : gbase;
    const size_t obase = CI ? cbase : (size_t)(bh / a.H) * a.out_sb + (size_t)h * a.out_sh;
    const Rows<D, CI> kr(a.k, base, m0, RS, L), vr(a.v, base, m0, RS, L), qr(a.q, base, m0, RS, L), dr(a.dout, obase, m0, OS, L);
    const float2* rs = reinterpret_cast<const float2*>(a.delta) + (size_t)bh * N + m0;
    auto stat_at = [&](int rows) {                       // of query row row_lo + rows
        unsigned long long x;
        asm("mad.wide.s32 %0, %1, 8, %2;" : "=l"(x) : "r"(rows), "l"(rs));
        return reinterpret_cast<const float2*>(x + 8u * (unsigned)g);
    };
    const float c2 = a.scale * kLog2e;
    const float gain = a.head_gain ? a.head_gain[h] : 1.f;

    RowFrag<D> ka, kb, va, vb;
    kr.template load2<AL>(ka, kb, 0, ok_lo, ok_hi);
    vr.template load2<AL>(va, vb, 0, ok_lo, ok_hi);
    float dK[D / 8][4], dV[D / 8][4];
    const float* se_lane = SE ? se_tile + 2 * tig * (kSeKeyPitch<WB> - 1) + WB + 16 + g : nullptr;

    // ---- dense window: query row of n-tile nt for this thread is m0 + 8 nt + g
    const __nv_bfloat16 *q_band = qr.at(0), *d_band = dr.at(0);
#pragma unroll
    for (int c = 0; c < NT / 2; ++c) {
        if (!INTERIOR && c > 0 && m0 + 16 * c >= N) break;   // warp-uniform: no query rows left
        RowFrag<D> qf[2], df[2];
        float ds[2][4], pv[2][4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int nt = 2 * c + hf;
            float s[4], dp[4];
            if constexpr (SE) {
                se_start_keys<WB>(s, se_lane, nt, g, tig);
            } else {
                StartTable<WB>::get(s, start, nt);
            }
            const __nv_bfloat16* qp = CI ? q_band + 8 * nt * D : qr.at(8 * nt);
            const __nv_bfloat16* dp_ = CI ? d_band + 8 * nt * D : dr.at(8 * nt);
            if (INTERIOR) {
                load_row_at<D, AL>(qf[hf], qp);
                load_row_at<D, AL>(df[hf], dp_);
            } else {
                const bool qv = m0 + 8 * nt + g < N;
                load_piece<D, AL>(qf[hf], qp, qv);
                load_piece<D, AL>(df[hf], dp_, qv);
            }
            mma_rows(s, ka, kb, qf[hf]);
            mma_rows_z(dp, va, vb, df[hf]);
            // statistics of this thread's two query columns: -l2 and -delta as pairs
            const f32x2 nl2 = *reinterpret_cast<const f32x2*>(stat_w + 8 * nt + 2 * tig);
            const f32x2 ndl = *reinterpret_cast<const f32x2*>(stat_w + kStat + 8 * nt + 2 * tig);
#pragma unroll
            for (int r = 0; r < 4; r += 2) {
                float p0, p1;
                unpair(fma2(pair(s[r], s[r + 1]), pair(c2, c2), nl2), p0, p1);
                p0 = ex2(p0); p1 = ex2(p1);
                pv[hf][r] = p0; pv[hf][r + 1] = p1;
                unpair(mul2(pair(p0, p1), fma2(pair(gain, gain), pair(dp[r], dp[r + 1]), ndl)), ds[hf][r], ds[hf][r + 1]);
            }
        }
        RowFrag<D> t0, t1;
        transpose_frag(t0, df[0]); transpose_frag(t1, df[1]);
        const uint32_t b0 = pack_bf16x2(pv[0][0], pv[0][1]), b1 = pack_bf16x2(pv[0][2], pv[0][3]);
        const uint32_t b2 = pack_bf16x2(pv[1][0], pv[1][1]), b3 = pack_bf16x2(pv[1][2], pv[1][3]);
        const uint32_t a0 = pack_bf16x2(ds[0][0], ds[0][1]), a1 = pack_bf16x2(ds[0][2], ds[0][3]);
        const uint32_t a2 = pack_bf16x2(ds[1][0], ds[1][1]), a3 = pack_bf16x2(ds[1][2], ds[1][3]);
        if (c == 0) {
#pragma unroll
            for (int j = 0; j < D / 8; ++j) mma16816_z(dV[j], b0, b1, b2, b3, t0.r[j], t1.r[j]);
        } else {
            mma_cols<D>(dV, b0, b1, b2, b3, t0, t1);
        }
        transpose_frag(t0, qf[0]); transpose_frag(t1, qf[1]);
        if (c == 0) {
#pragma unroll
            for (int j = 0; j < D / 8; ++j) mma16816_z(dK[j], a0, a1, a2, a3, t0.r[j], t1.r[j]);
        } else {
            mma_cols<D>(dK, a0, a1, a2, a3, t0, t1);
        }
    }
    // ---- sparse taps
    const int ns8 = (ns + 7) / 8 * 8;
    const float* qs_r = SE ? a.qs_rows + ((size_t)bh * N + row_lo) * ns8 : nullptr;   // entry of tap si of query row row_lo + delta: qs_r[delta * ns8 + si]
    // b0/b1: what is added to the raw score: the bias in log2 units (plain) or the qs_rows entry of
    // the query row, in units of 1/scale (scale_embed)
    auto finish = [&](float sd0, float sd1, float dp0, float dp1, float b0, float b1, float2 st0, float2 st1,
                      const RowFrag<D>& qf0, const RowFrag<D>& qf1, const RowFrag<D>& df0, const RowFrag<D>& df1) {
        const float y0 = SE ? (sd0 + b0) * c2 : fmaf(sd0, c2, b0), y1 = SE ? (sd1 + b1) * c2 : fmaf(sd1, c2, b1);
        const float p0 = ex2(y0 - st0.x), p1 = ex2(y1 - st1.x);
        const float x0 = p0 * fmaf(gain, dp0, -st0.y), x1 = p1 * fmaf(gain, dp1, -st1.y);
        diag_fma<D>(dV, __shfl_sync(0xffffffffu, p0, L.owner_lane), __shfl_sync(0xffffffffu, p1, L.owner_lane), df0, df1);
        diag_fma<D>(dK, __shfl_sync(0xffffffffu, x0, L.owner_lane), __shfl_sync(0xffffffffu, x1, L.owner_lane), qf0, qf1);
    };
    auto full_taps = [&](auto GC, int si) {
        constexpr int GG = decltype(GC)::value;
        RowFrag<D> qf0[GG], qf1[GG], df0[GG], df1[GG];
        float2 st0[GG], st1[GG];
        float b0[GG], b1[GG];
#pragma unroll
        for (int i = 0; i < GG; ++i) {
            const int2 tp = make_int2(t.sparse[si + i], tap_s[si + i].y);
            if constexpr (SE) {
                b0[i] = __ldg(qs_r + (size_t)tp.x * ns8 + si + i);
                b1[i] = __ldg(qs_r + (size_t)(tp.x + 8) * ns8 + si + i);
            } else {
                b0[i] = b1[i] = __int_as_float(tp.y);
            }
            qr.template load2<AL>(qf0[i], qf1[i], tp.x);
            dr.template load2<AL>(df0[i], df1[i], tp.x);
            const float2* st = stat_at(tp.x);
            st0[i] = __ldg(st);
            st1[i] = __ldg(st + 8);
        }
#pragma unroll
        for (int i = 0; i < GG; ++i) {
            float s0[4], s1[4], e0[4], e1[4];
            mma_rows_z(s0, ka, kb, qf0[i]); mma_rows_z(s1, ka, kb, qf1[i]);
            mma_rows_z(e0, va, vb, df0[i]); mma_rows_z(e1, va, vb, df1[i]);
            finish((g & 1) ? s0[1] : s0[0], (g & 1) ? s1[3] : s1[2], (g & 1) ? e0[1] : e0[0], (g & 1) ? e1[3] : e1[2],
                   b0[i], b1[i], st0[i], st1[i], qf0[i], qf1[i], df0[i], df1[i]);
        }
    };
    int si = 0;
    for (; si + G <= ns && m0 + 16 + t.sparse[si + G - 1] <= N; si += G) full_taps(std::integral_constant<int, G>(), si);
#pragma unroll 1
    for (; si < ns; ++si) {
        const int delta = t.sparse[si];
        if (m0 + delta >= N) break;                     // taps ascend: no query row reads these keys any more
        if (m0 + 16 + delta <= N) {
            full_taps(std::integral_constant<int, 1>(), si);
        } else {
            const bool v0 = row_lo + delta < N, v1 = row_hi + delta < N;
            float b0 = __int_as_float(tap_s[si].y), b1 = b0;
            if constexpr (SE) {
                b0 = v0 ? __ldg(qs_r + (size_t)delta * ns8 + si) : 0.f;
                b1 = v1 ? __ldg(qs_r + (size_t)(delta + 8) * ns8 + si) : 0.f;
            }
            RowFrag<D> qf0, qf1, df0, df1;
            qr.template load2<AL>(qf0, qf1, delta, v0, v1);
            dr.template load2<AL>(df0, df1, delta, v0, v1);
            const float2* st = stat_at(delta);
            const float2 st0 = v0 ? __ldg(st) : make_float2(0.f, 0.f);
            const float2 st1 = v1 ? __ldg(st + 8) : make_float2(0.f, 0.f);
            float s0[4], s1[4], e0[4], e1[4];
            mma_rows_z(s0, ka, kb, qf0); mma_rows_z(s1, ka, kb, qf1);
            mma_rows_z(e0, va, vb, df0); mma_rows_z(e1, va, vb, df1);
            finish((g & 1) ? s0[1] : s0[0], (g & 1) ? s1[3] : s1[2], (g & 1) ? e0[1] : e0[0], (g & 1) ? e1[3] : e1[2],
                   b0, b1, st0, st1, qf0, qf1, df0, df1);
        }
    }
    __nv_bfloat16* dkp = static_cast<__nv_bfloat16*>(a.dk) + gbase;
    __nv_bfloat16* dvp = static_cast<__nv_bfloat16*>(a.dv) + gbase;
    store_acc_rows<D, AL>(dK, dkp + (size_t)row_lo * GS, dkp + (size_t)row_hi * GS, ok_lo, ok_hi, a.scale, a.scale, tig);
    store_acc_rows<D, AL>(dV, dvp + (size_t)row_lo * GS, dvp + (size_t)row_hi * GS, ok_lo, ok_hi, gain, gain, tig);   // dV = gain P^T.dO
}

template <int WB> inline size_t dkdv_smem_bytes(bool se) { return se ? (size_t)(kRows + WB) * kSeKeyPitch<WB> * 4 : 0; }

template <int D, int WB, int G, int CT, bool SE, int ST>
__global__ void __launch_bounds__(kWarps * 32, CT)
bwd_dkdv_mma_kernel(const BwdArgs a, const Taps t, const int n_reduce, const int reduce_stride) {
    stream_wait();
    constexpr int kStat = kRows + WB;                  // query rows the CTA's dense windows touch
    extern __shared__ __align__(16) float se_tile[];   // scale_embed: [kStat][kSeKeyPitch]
    __shared__ __align__(16) float start_s[SE ? 4 : StartTable<WB>::kSize];
    __shared__ float red_s[kReduceThreads];
    __shared__ int2 tap_s[DSQG_MAX_TAPS];
    __shared__ __align__(16) float stat_s[2 * kStat];  // -lse * log2(e) of the rows, then -delta
    const Lane L;
    const int bh = blockIdx.y, h = bh % a.H, N = a.N;
    // Every reduce_stride-th CTA (so that no wave of CTAs is delayed as a whole) also finishes the
    // parameter gradients: n_reduce outputs in all, from the partial sums the dQ kernel (an earlier
    // launch on the stream) left in the scratch.
    static_assert(kWarps * 32 == kReduceThreads, "the fused reduction uses the CTA as one reduce block");
    const int cta = blockIdx.y * gridDim.x + blockIdx.x;
    if (cta % reduce_stride == 0)
        for (int o = cta / reduce_stride; o < n_reduce; o += gridDim.x * gridDim.y / reduce_stride)
            reduce_one_param(a, t.J, o, red_s);
    const int m_cta = blockIdx.x * kRows;
    {
        if constexpr (!SE) StartTable<WB>::template fill<true, kWarps * 32>(start_s, a.pos_bias, a.H, h, t.d_lo, t.d_lo + t.n_dense - 1, a.scale);
        for (int si = threadIdx.x; si < t.n_sparse; si += kWarps * 32)
            tap_s[si] = make_int2(t.sparse[si], __float_as_int(a.pos_bias[(t.n_dense + si) * a.H + h] * kLog2e));
        const float2* rs = reinterpret_cast<const float2*>(a.delta) + (size_t)bh * N;
        for (int i = threadIdx.x; i < kStat; i += kWarps * 32) {
            const float2 x = m_cta + i < N ? rs[m_cta + i] : make_float2(0.f, 0.f);
            stat_s[i] = -x.x; stat_s[kStat + i] = -x.y;
        }
        if constexpr (SE) {
            const SePre P = se_pre_layout<WB>(a.se_pre, t.n_sparse, D);
            const SeRows rows = {P.hi, P.lo, P.pb + h * SeGeo<WB>::rows(t.n_sparse)};
            constexpr bool AL = ST != kStridedAny, CI = ST == kContiguous || ST == kKept;
            const ptrdiff_t RS = CI ? D : (ptrdiff_t)a.in_sn;
            const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(a.q) + (CI ? (size_t)bh * N * D : (size_t)(bh / a.H) * a.in_sb + (size_t)h * a.in_sh);
#pragma unroll 1
            for (int b = L.warp; b < kStat / 16; b += kWarps) {
                const int r = m_cta + 16 * b + L.g;
                RowFrag<D> qa, qb;
                load_row<D, AL>(qa, q + (ptrdiff_t)r * RS, L.tig, r < N);
                load_row<D, AL>(qb, q + (ptrdiff_t)(r + 8) * RS, L.tig, r + 8 < N);
                build_se_tile<D, WB, true>(rows, 0, qa, qb, L.g, L.tig, se_tile + 16 * b * kSeKeyPitch<WB>, kSeKeyPitch<WB>, nullptr, 0);
            }
        }
    }
    __syncthreads();
    const int m0 = m_cta + L.warp * 16;
    if (m0 >= N) return;
    const float* se_w = SE ? se_tile + L.warp * 16 * kSeKeyPitch<WB> : nullptr;
    const float* start = StartTable<WB>::lane(start_s, L);
    if (m0 + 16 + WB <= N)
        dkdv_tile<D, WB, true, G, SE, ST>(a, start, tap_s, stat_s + L.warp * 16, t, t.n_sparse, bh, h, m0, L, se_w);
    else
        dkdv_tile<D, WB, false, G, SE, ST>(a, start, tap_s, stat_s + L.warp * 16, t, t.n_sparse, bh, h, m0, L, se_w);
}

// Raises a kernel's dynamic shared-memory limit to what this launch needs.  The attribute is set
// once per kernel and device for the largest size seen so far (`seen` is that kernel's record),
// not on every launch.
template <typename K>
cudaError_t ensure_dynamic_smem(K kernel, size_t bytes, int (&seen)[64]) {
    if (bytes <= 32 * 1024) return cudaSuccess;        // static shared memory counts against the 48 KB default as well
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && seen[dev] >= (int)bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && dev >= 0 && dev < 64) seen[dev] = (int)bytes;
    return e;
}

// Whether every piece of every row starts on a multiple of `bytes`.
inline bool aligned_to(size_t bytes, std::initializer_list<const void*> ptrs, std::initializer_list<long long> strides) {
    for (const void* p : ptrs) if (reinterpret_cast<uintptr_t>(p) % bytes) return false;
    for (long long x : strides) if ((size_t)x * 2 % bytes) return false;
    return true;
}

template <int D, int WB, bool SE, int ST>
cudaError_t fwd_launch_mode(const FwdArgs& a, const Taps& t, cudaStream_t s) {
    constexpr int W = FwdTune<D>::warps;
    const int tiles_se = SE ? FwdTune<D>::tiles_se(a.N, a.B * a.H) : 1, rows = 16 * W * tiles_se;
    dim3 grid((a.N + rows - 1) / rows, a.B * a.H);
    size_t smem = 0;
    if constexpr (SE) {
        static int seen[64] = {0};
        smem = se_rows_bytes<WB>(t.n_sparse, D) + W * se_tile_floats<WB>(t.n_sparse) * 4;
        const cudaError_t e = ensure_dynamic_smem(fwd_mma_kernel<D, WB, SE, ST>, smem, seen);
        if (e != cudaSuccess) return e;
    }
    return launch_after(fwd_mma_kernel<D, WB, SE, ST>, grid, W * 32, smem, s, a, t, tiles_se);
}

template <int D, int WB, bool SE>
cudaError_t fwd_launch_se(FwdArgs a, const Taps& t, cudaStream_t s) {
    if constexpr (kLane<D> == 16) {       // 32-byte pieces
        if (!aligned_to(32, {a.q, a.k, a.v, a.out, a.gate, a.keep}, {a.in_sb, a.in_sh, a.in_sn, a.out_sb, a.out_sh, a.out_sn, a.gate_sb, a.gate_sh, a.gate_sn})) {
            if (!a.strided) {
                a.in_sn = a.out_sn = D; a.in_sh = a.out_sh = (long long)a.N * D; a.in_sb = a.out_sb = (long long)a.H * a.N * D;
            }
            return fwd_launch_mode<D, WB, SE, kStridedAny>(a, t, s);
        }
    }
    if (!a.strided) return fwd_launch_mode<D, WB, SE, kContiguous>(a, t, s);
    if constexpr (kTail<D>) return cudaErrorInvalidValue;
    else return fwd_launch_mode<D, WB, SE, kStrided>(a, t, s);
}

template <int D, int WB>
cudaError_t fwd_launch_mma(const FwdArgs& a, const Taps& t, cudaStream_t s) {
    if (!a.scale_embed) return fwd_launch_se<D, WB, false>(a, t, s);
    if constexpr (D <= 64 && !kTail<D>) return fwd_launch_se<D, WB, true>(a, t, s);
    else return cudaErrorInvalidValue;
}

template <int D, int WB, bool SE, int ST>
cudaError_t bwd_launch_mode(BwdArgs a, const Taps& t, cudaStream_t s, int stages) {
    using T = BwdTune<D>;
    if constexpr (SE) carve_bwd_scratch_mma_se(a, t.J); else carve_bwd_scratch(a, kRows, t.J, false);
    dim3 grid((a.N + kRows - 1) / kRows, a.B * a.H);
    cudaError_t e = cudaSuccess;
    if (stages & DSQG_BWD_STAGE_DQ) {
        if constexpr (SE) {
            if ((e = launch_after(se_prep_kernel<D, WB>, 1, 1024, 0, s, a.scale_embed, a.pos_bias, a.scale, t, a.H, a.se_pre)) != cudaSuccess) return e;
        }
        auto kern = bwd_dq_mma_kernel<D, WB, SE ? T::dq_group_se : T::dq_group, SE ? T::dq_ctas_se : T::dq_ctas, SE, ST>;
        const size_t smem = dq_smem_bytes<D, WB>(t.J, t.n_sparse, SE);
        static int seen[64] = {0};
        if ((e = ensure_dynamic_smem(kern, smem, seen)) != cudaSuccess) return e;
        if ((e = launch_after(kern, grid, kWarps * 32, smem, s, a, t)) != cudaSuccess) return e;
        if constexpr (SE) {
            const int groups_bh = (a.tiles_per_bh + kSeGroup - 1) / kSeGroup;
            if ((e = launch_after(dse_group_kernel, dim3(groups_bh, a.B * a.H), 256, 0, s, a.dse_tmp, a.dse_part, a.tiles_per_bh, groups_bh, t.J * a.D)) != cudaSuccess) return e;
        }
    }
    // With both stages in one call the reduction rides on CTAs of the dK/dV kernel (same code,
    // same order of additions as the stand-alone kernel: bitwise equal results).  Up to four outputs per
    // CTA cost less than the launch they save (about 1 us each against 2.7 us on the GPU and 4 us on the host).
    const int n_out = t.J * a.H + a.H + (SE ? t.J * a.D : 0);
    const bool fuse = (stages & DSQG_BWD_STAGE_DKDV) && (stages & DSQG_BWD_STAGE_REDUCE) &&
                      4LL * grid.x * grid.y >= n_out;
    if (stages & DSQG_BWD_STAGE_DKDV) {
        auto kern = bwd_dkdv_mma_kernel<D, WB, SE ? T::dkdv_group_se : T::dkdv_group, SE ? T::dkdv_ctas_se : T::dkdv_ctas, SE, ST>;
        const size_t smem = dkdv_smem_bytes<WB>(SE);
        static int seen[64] = {0};
        if ((e = ensure_dynamic_smem(kern, smem, seen)) != cudaSuccess) return e;
        e = launch_after(kern, grid, kWarps * 32, smem, s, a, t, fuse ? n_out : 0, fuse && (long long)grid.x * grid.y >= n_out ? (int)((long long)grid.x * grid.y / n_out) : 1);
        if (e != cudaSuccess) return e;
    }
    if ((stages & DSQG_BWD_STAGE_REDUCE) && !fuse) e = launch_reduce_params(a, t.J, s);
    return e;
}

template <int D, int WB, bool SE>
cudaError_t bwd_launch_se(BwdArgs a, const Taps& t, cudaStream_t s, int stages) {
    // A gate that starts on 16 bytes only takes both kernels along: packed backward 16x12x2048x64 326.5 us against 297.0 (337.6 wherever it started when it
    // had a kernel of its own ahead of these), 8x8x2048x128 267.7 against 248.5 (267.4).
    if constexpr (kLane<D> == 16) {       // 32-byte pieces
        if (!aligned_to(32, {a.q, a.k, a.v, a.out, a.dout, a.dq, a.dk, a.dv, a.dy, a.y, a.gate, a.dgate}, {a.in_sb, a.in_sh, a.in_sn, a.out_sb, a.out_sh, a.out_sn}) ||
            (a.gate && !aligned_to(32, {}, {a.y_st.batch, a.y_st.head, a.y_st.row, a.gate_st.batch, a.gate_st.head, a.gate_st.row, a.dgate_st.batch, a.dgate_st.head, a.dgate_st.row}))) {
            if (!a.strided) {
                a.in_sn = a.out_sn = D; a.in_sh = a.out_sh = (long long)a.N * D; a.in_sb = a.out_sb = (long long)a.H * a.N * D;
            }
            return bwd_launch_mode<D, WB, SE, kStridedAny>(a, t, s, stages);
        }
    }
    if (!a.strided) return bwd_launch_mode<D, WB, SE, kContiguous>(a, t, s, stages);
    if (a.kept) {
        if constexpr (kept_pays(D)) return bwd_launch_mode<D, WB, SE, kKept>(a, t, s, stages);
        else return cudaErrorInvalidValue;
    }
    if constexpr (kTail<D>) return cudaErrorInvalidValue;
    else return bwd_launch_mode<D, WB, SE, kStrided>(a, t, s, stages);
}

template <int D, int WB>
cudaError_t bwd_launch_mma(const BwdArgs& a, const Taps& t, cudaStream_t s, int stages) {
    if (!a.scale_embed) return bwd_launch_se<D, WB, false>(a, t, s, stages);
    if constexpr (D <= 64 && !kTail<D>) return bwd_launch_se<D, WB, true>(a, t, s, stages);
    else return cudaErrorInvalidValue;
}

inline int band_width(const Taps& t) {
    const int d_hi = t.d_lo + t.n_dense - 1;
    return d_hi <= 32 ? 32 : (d_hi <= 48 ? 48 : (d_hi <= 64 ? 64 : 0));
}

}  // namespace

}  // namespace dsqg
