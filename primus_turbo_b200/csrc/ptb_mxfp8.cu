// MXFP8 quantise / dequantise for sm_100a: 1x32 (or 32x32) blocks with power-of-two E8M0 scales.
//
// Semantics follow the reference's csrc/kernels/quantization/quantization_mxfp8.cu (scale from the block
// maximum: lines 71-110; 32x32 tiles, zero fill outside the matrix, clamp to +-(fmax * scale) then divide
// by the scale: lines 128-515) and dequantization_mxfp8.cu:47-100.  Layouts follow
// csrc/pytorch/quantization/quantization.cpp:736-966: the row-direction output is [M, N_pad], the
// column-direction output is stored TRANSPOSED as [N, M_pad], padded extents are multiples of 128 and
// hold zero bytes with scale byte 0, scales are one byte per 32 elements along the padded extent.
//
// One pass over the input produces both directions.  A warp owns a 32-row x 64-column tile and never
// talks to another warp: row maxima reduce over the four lanes of a 32-column block, column maxima over
// the four lanes that share a column, and the transposed output is assembled with a 4x4 byte transpose
// across those four lanes, so every lane ends up holding 32 contiguous output bytes of two columns.
#include "ptb_common.cuh"

// resident CTAs per SM the quantise kernel is compiled for (85 registers a thread at three)
#ifndef PTB_MXQ_MINB
#define PTB_MXQ_MINB 3
#endif

namespace ptb {
namespace {

constexpr int kMxBlock = 32;
constexpr int kMxPad   = 128;

template <int FMT> struct MxFmt;
template <> struct MxFmt<PTB_E4M3> { static constexpr int mbits = 3, target_pow2 = 8; };
template <> struct MxFmt<PTB_E5M2> { static constexpr int mbits = 2, target_pow2 = 15; };

// Block maximum -> biased E8M0 byte.  The maximum's mantissa is rounded to the FP8 format's width (the
// carry may bump the exponent), the exponent of the format's largest power of two is subtracted, the
// result is clamped to [-127, 128] and biased by 127.  A maximum is never negative, never NaN and at most infinity, so the biased
// exponent before the subtraction is at most 255 and only the lower clamp can bind.
template <int FMT, bool ZERO_IS_ONE> __device__ __forceinline__ int mx_byte(float amax) {
    if (ZERO_IS_ONE && amax == 0.0f) return 127;
    constexpr uint32_t add = 1u << (23 - MxFmt<FMT>::mbits - 1);
    return max((int) ((__float_as_uint(amax) + add) >> 23) - MxFmt<FMT>::target_pow2, 0);
}
// The reference clamps a value to +-(fmax * scale), scale = (byte << 23) read as fp32, and divides by the
// scale.  Here: multiply by the exact reciprocal 2^(127 - byte) (bytes stay below 248, so it is a normal number) and let
// the saturating conversion clamp -- the same result for every finite value, because fmax * scale times the
// reciprocal is exactly fmax.  Byte 0 is the one exception: its scale reads as 0.0f, the clamp limit is zero
// and every value becomes +-0, which a multiplier of zero reproduces (sign included).
__device__ __forceinline__ float mx_inverse(int biased) {
    return biased == 0 ? 0.0f : __uint_as_float((uint32_t) (254 - biased) << 23);
}

struct MxQuantArgs {
    const void *x;
    uint8_t *q_row, *s_row, *q_col, *s_col;
    int64_t M, N, M_pad, N_pad;
    int row_2d, col_2d;
    // grouped mode: per 128-row block of the padded column layout {first source row, end of the group's
    // source rows, row of the row-direction output that the first source row goes to, group}
    const int4 *table;
};

// Grouped layouts (csrc/pytorch/quantization/quantization.cpp:1100-1130 in the reference): every group's rows
// padded to `row_align` rows in the row-direction output and to 128 rows in the column-direction output.
// One CTA: padded lengths and offsets of both layouts and the block table of MxQuantArgs; blocks past the
// last group get an empty entry (they are written as zeros).
__global__ void __launch_bounds__(256) mx_group_layout_kernel(const int64_t *group_offs, int64_t G, int64_t row_align,
                                                              int64_t *row_lens, int64_t *row_offs,
                                                              int64_t *col_lens, int64_t *col_offs,
                                                              int4 *table, int64_t nblocks) {
    grid_dep_begin();
    __shared__ int64_t s_row[256], s_col[256];
    const int tid     = threadIdx.x;
    const int64_t per = cdiv<int64_t>(G, 256);
    const int64_t g0 = (int64_t) tid * per, g1 = imin(g0 + per, G);
    int64_t lr = 0, lc = 0;
    for (int64_t g = g0; g < g1; ++g) {
        const int64_t len = group_offs[g + 1] - group_offs[g];
        lr += cdiv<int64_t>(len, row_align) * row_align;
        lc += cdiv<int64_t>(len, kMxPad) * kMxPad;
    }
    s_row[tid] = lr;
    s_col[tid] = lc;
    __syncthreads();
    for (int off = 1; off < 256; off <<= 1) {
        const int64_t ar = (tid >= off) ? s_row[tid - off] : 0, ac = (tid >= off) ? s_col[tid - off] : 0;
        __syncthreads();
        s_row[tid] += ar;
        s_col[tid] += ac;
        __syncthreads();
    }
    int64_t run_r = s_row[tid] - lr, run_c = s_col[tid] - lc;
    for (int64_t g = g0; g < g1; ++g) {
        const int64_t gs = group_offs[g], ge = group_offs[g + 1];
        const int64_t pr = cdiv<int64_t>(ge - gs, row_align) * row_align, pc = cdiv<int64_t>(ge - gs, kMxPad) * kMxPad;
        row_lens[g] = pr; row_offs[g] = run_r;
        col_lens[g] = pc; col_offs[g] = run_c;
        for (int64_t t = 0; t < pc / kMxPad; ++t)
            table[run_c / kMxPad + t] = make_int4((int) (gs + t * kMxPad), (int) ge, (int) (run_r + t * kMxPad), (int) g);
        run_r += pr;
        run_c += pc;
    }
    if (tid == 255) { row_offs[G] = s_row[255]; col_offs[G] = s_col[255]; }
    for (int64_t b = s_col[255] / kMxPad + tid; b < nblocks; b += 256) table[b] = make_int4(0, 0, 0, -1);
}

// column tiles one CTA walks (16384 x 8192 bf16, both directions: one tile per CTA 0.176 ms, strips of two
// 0.162 ms, of four 0.148 ms)
#ifndef PTB_MX_STRIP
#define PTB_MX_STRIP 4
#endif
constexpr int kMxStrip = PTB_MX_STRIP;
__device__ __forceinline__ void mx_cp_async16_zfill(void *dst_smem, const void *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t) __cvta_generic_to_shared(dst_smem)), "l"(src),
                 "r"(valid ? 16u : 0u)
                 : "memory");
}

template <typename T> struct Pair;
template <> struct Pair<__nv_bfloat16> {
    using type = __nv_bfloat162;
    static __device__ __forceinline__ float2 f2(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<const type *>(&v)); }
};
template <> struct Pair<__half> {
    using type = __half2;
    static __device__ __forceinline__ float2 f2(uint32_t v) { return __half22float2(*reinterpret_cast<const type *>(&v)); }
};
// two 16-bit values an instruction; magnitudes and maxima are exact
template <typename T> __device__ __forceinline__ uint32_t abs2(uint32_t a) {
    using T2 = typename Pair<T>::type;
    const T2 r = __habs2(*reinterpret_cast<const T2 *>(&a));
    return *reinterpret_cast<const uint32_t *>(&r);
}
template <typename T> __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    using T2 = typename Pair<T>::type;
    const T2 r = __hmax2(*reinterpret_cast<const T2 *>(&a), *reinterpret_cast<const T2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}
template <typename T> __device__ __forceinline__ uint32_t shfl_max2(uint32_t a, int lanes) {
    return max2<T>(a, __shfl_xor_sync(0xffffffffu, a, lanes));
}
// four values (two packed words) times their scales -> four FP8 bytes
template <typename T, int FMT> __device__ __forceinline__ uint32_t mx_cvt4(uint32_t lo, uint32_t hi, float2 s_lo, float2 s_hi) {
    const float2 a = __fmul2_rn(Pair<T>::f2(lo), s_lo), b = __fmul2_rn(Pair<T>::f2(hi), s_hi);
    return (uint32_t) cvt_fp8x2<FMT>(a.x, a.y) | ((uint32_t) cvt_fp8x2<FMT>(b.x, b.y) << 16);
}
__device__ __forceinline__ void store_scale_word(uint8_t *dst, uint32_t w) {
    if ((reinterpret_cast<uintptr_t>(dst) & 3u) == 0) {
        *reinterpret_cast<uint32_t *>(dst) = w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = (uint8_t) (w >> (8 * i));
    }
}

// grid: (ceil(N_pad / 128 / kMxStrip), M_pad / 128, G); 256 threads; warp w: rows 32 * (w & 3), columns 64 * (w >> 2) of a tile
// GROUPED: blockIdx.y walks the 128-row blocks of the padded column layout; the block table says which
// source rows it holds and where they go in the row-direction output; a block maximum of zero takes scale
// byte 127 (1.0) instead of 0, as the reference's grouped kernel does (quantization_mxfp8.cu:1425-1450).
//
// Bound by HBM (4 bytes an element) once the instruction and transaction counts allow it.  Maxima stay packed in 16 bits, two
// rows or columns a word, which halves the maximum and shuffle instructions and lets three CTAs of the SM share the
// registers; scale bytes meet in shared memory and leave as 4-byte words at the end of the strip (a byte a store
// was as many L2 transactions as the column copy itself); a column's 32 bytes leave in one store.  32 x 4096 x 7168
// bf16, both directions: 976 -> 625 us; grouped activations of 8192 rows, 7168 and 4096 wide: 205 -> 96 us.
template <typename T, int FMT, bool GROUPED>
__global__ void __launch_bounds__(256, PTB_MXQ_MINB) mx_quant_kernel(const MxQuantArgs p) {
    grid_dep_begin();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rl = lane >> 3, cl = lane & 7;
    const int wr = warp & 3, wc = warp >> 2;
    const int64_t g    = GROUPED ? 0 : blockIdx.z;
    const int64_t row0 = (int64_t) blockIdx.y * 128 + 32 * wr; // row of the (padded) column layout
    const T *x         = reinterpret_cast<const T *>(p.x) + g * p.M * p.N;
    // first source row of this CTA, end of valid rows, row-output row of the first source row
    int64_t src_blk = (int64_t) blockIdx.y * 128, src_end = p.M, out_blk = src_blk;
    if constexpr (GROUPED) {
        const int4 e = p.table[blockIdx.y];
        src_blk      = e.x;
        src_end      = e.y;
        out_blk      = e.z;
    }
    const int64_t src0 = src_blk + 32 * wr + rl; // this lane's first row (then every fourth)
    const int rows_left = (int) imin(32, imax(0, src_end - src0)); // rows src0, src0 + 4, ... that exist: 4 ps < rows_left

    // A CTA walks kMxStrip consecutive column tiles; the fragments of the tile after the current one are already
    // on their way (cp.async into this thread's own shared-memory slots, zero-filled outside the matrix).
    __shared__ uint4 s_frag[8][256];
    __shared__ __align__(4) uint8_t s_rowb[128][4 * kMxStrip + 4]; // scale bytes of the strip; rows padded by a bank
    __shared__ __align__(4) uint8_t s_colb[128 * kMxStrip][4];
    const int tiles_x = (int) (p.N_pad / 128);
    const int tx0     = (int) blockIdx.x * kMxStrip;
    const int ntiles  = min(kMxStrip, tiles_x - tx0);
    auto issue = [&](int t) {
        const int64_t c = (int64_t) (tx0 + t) * 128 + 64 * wc + cl * 8;
        const T *src    = x + src0 * p.N + c;
#pragma unroll
        for (int ps = 0; ps < 8; ++ps) {
            const bool valid = 4 * ps < rows_left && c < p.N;
            mx_cp_async16_zfill(&s_frag[ps][threadIdx.x], valid ? (const void *) (src + 4 * ps * p.N) : (const void *) x, valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0);
    for (int t = 0; t < ntiles; ++t) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        uint4 raw[8];
#pragma unroll
        for (int ps = 0; ps < 8; ++ps) raw[ps] = s_frag[ps][threadIdx.x];
        if (t + 1 < ntiles) issue(t + 1);
        const int64_t col = (int64_t) (tx0 + t) * 128 + 64 * wc + cl * 8;
        // cm[i]: maxima of columns 2 i, 2 i + 1 over the warp's 32 rows; rm[i]: of rows 2 i, 2 i + 1 (of this lane's eight)
        // over the 32-column block
        uint32_t cm[4] = {0, 0, 0, 0}, rm[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t m[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint4 &r = raw[2 * i + k];
                const uint32_t a0 = abs2<T>(r.x), a1 = abs2<T>(r.y), a2 = abs2<T>(r.z), a3 = abs2<T>(r.w);
                cm[0] = max2<T>(cm[0], a0);
                cm[1] = max2<T>(cm[1], a1);
                cm[2] = max2<T>(cm[2], a2);
                cm[3] = max2<T>(cm[3], a3);
                m[k]  = max2<T>(max2<T>(a0, a1), max2<T>(a2, a3));
            }
            // from zero, like the column maxima: a maximum passes over NaN also where a lane holds nothing else
            const uint32_t both = max2<T>(max2<T>(0u, __byte_perm(m[0], m[1], 0x5410)), __byte_perm(m[0], m[1], 0x7632));
            rm[i]               = shfl_max2<T>(shfl_max2<T>(both, 1), 2); // the four lanes of a 32-column block
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) cm[i] = shfl_max2<T>(shfl_max2<T>(cm[i], 8), 16); // the four lanes that share a column
        if (p.row_2d || p.col_2d) { // one maximum per 32x32 tile: every row / column of it takes that one
            uint32_t m = max2<T>(max2<T>(cm[0], cm[1]), max2<T>(cm[2], cm[3]));
            m          = shfl_max2<T>(shfl_max2<T>(m, 1), 2);
            m          = max2<T>(m, __byte_perm(m, m, 0x1032));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (p.row_2d) rm[i] = m;
                if (p.col_2d) cm[i] = m;
            }
        }

        // ---- row direction: q_row[g][r][col .. col+7], s_row[g][r][col / 32] -----------------------------
        if (p.q_row != nullptr) {
            uint8_t *q = p.q_row + (g * p.M + out_blk + 32 * wr + rl) * p.N_pad + col;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 m = Pair<T>::f2(rm[i]);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int ps = 2 * i + k;
                    if (4 * ps >= rows_left) continue; // only rows that exist are written
                    const int biased = mx_byte<FMT, GROUPED>(k ? m.y : m.x);
                    const float inv  = mx_inverse(biased);
                    const float2 s2  = make_float2(inv, inv);
                    *reinterpret_cast<uint2 *>(q + 4 * ps * p.N_pad) =
                        make_uint2(mx_cvt4<T, FMT>(raw[ps].x, raw[ps].y, s2, s2), mx_cvt4<T, FMT>(raw[ps].z, raw[ps].w, s2, s2));
                    if ((cl & 3) == 0) s_rowb[32 * wr + 4 * ps + rl][4 * t + 2 * wc + (cl >> 2)] = (uint8_t) biased;
                }
            }
        }

        // ---- column direction: q_col[g][c][row0 .. row0+31] (transposed), s_col[g][c][row0 / 32] ---------
        if (p.q_col != nullptr) {
            uint8_t *q = p.q_col + g * p.N * p.M_pad;
            // two passes of four columns each keep the live state small
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 m01 = Pair<T>::f2(cm[2 * h]), m23 = Pair<T>::f2(cm[2 * h + 1]);
                const int b0 = mx_byte<FMT, GROUPED>(m01.x), b1 = mx_byte<FMT, GROUPED>(m01.y);
                const int b2 = mx_byte<FMT, GROUPED>(m23.x), b3 = mx_byte<FMT, GROUPED>(m23.y);
                const float2 s01 = make_float2(mx_inverse(b0), mx_inverse(b1)), s23 = make_float2(mx_inverse(b2), mx_inverse(b3));
                // lane rl writes the byte of column 4 h + rl
                s_colb[128 * t + 64 * wc + cl * 8 + 4 * h + rl][wr] = (uint8_t) (rl < 2 ? (rl == 0 ? b0 : b1) : (rl == 2 ? b2 : b3));
                // w[ps]: this lane's row (4 ps + rl), columns 4 h .. 4 h + 3, one byte each
                uint32_t w[8];
#pragma unroll
                for (int ps = 0; ps < 8; ++ps)
                    w[ps] = h == 0 ? mx_cvt4<T, FMT>(raw[ps].x, raw[ps].y, s01, s23) : mx_cvt4<T, FMT>(raw[ps].z, raw[ps].w, s01, s23);
                // 4x4 byte transpose across the lanes rl = 0..3 (lane bits 3 and 4): afterwards byte k of
                // w[ps] is row 4 ps + k of column 4 h + rl
#pragma unroll
                for (int ps = 0; ps < 8; ++ps) {
                    uint32_t mine  = w[ps];
                    uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 8);
                    mine           = __byte_perm(mine, other, (rl & 1) ? 0x3715 : 0x6240);
                    other          = __shfl_xor_sync(0xffffffffu, mine, 16);
                    mine           = __byte_perm(mine, other, (rl & 2) ? 0x3276 : 0x5410);
                    w[ps]          = mine;
                }
                const int64_t c = col + 4 * h + rl;
                if (c < p.N) {
                    uint8_t *dst = q + c * p.M_pad + row0; // row0 and M_pad are multiples of 32
                    if ((reinterpret_cast<uintptr_t>(p.q_col) & 31u) == 0) {
                        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]),
                                     "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                                     : "memory");
                    } else {
                        reinterpret_cast<uint4 *>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                        reinterpret_cast<uint4 *>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                    }
                }
            }
        }
    } // column tiles of the strip

    // ---- scale bytes of the strip: four columns' blocks, or four row blocks, per word -----------------------
    __syncthreads();
    if (p.q_row != nullptr) {
        const int64_t pitch = p.N_pad / kMxBlock;
        uint8_t *s          = p.s_row + (g * p.M + out_blk) * pitch + (int64_t) tx0 * 4;
        for (int i = threadIdx.x; i < 128 * kMxStrip; i += 256) {
            const int r = i / kMxStrip, t = i % kMxStrip;
            if (t < ntiles && src_blk + r < src_end)
                store_scale_word(s + r * pitch + 4 * t, *reinterpret_cast<const uint32_t *>(&s_rowb[r][4 * t]));
        }
    }
    if (p.q_col != nullptr) {
        const int64_t pitch = p.M_pad / kMxBlock;
        uint8_t *s          = p.s_col + (g * p.N + (int64_t) tx0 * 128) * pitch + (int64_t) blockIdx.y * 4;
        for (int i = threadIdx.x; i < 128 * ntiles; i += 256)
            if ((int64_t) tx0 * 128 + i < p.N) store_scale_word(s + i * pitch, *reinterpret_cast<const uint32_t *>(s_colb[i]));
    }
}

// out[r][c] = cast(float(q[r][c]) * (scale byte << 23 read as fp32)); TRANSPOSE writes out[c][r] instead
template <typename TO, int FMT, bool TRANSPOSE>
__global__ void __launch_bounds__(256) mx_dequant_kernel(const uint8_t *__restrict__ q, const uint8_t *__restrict__ s,
                                                         int64_t R, int64_t C, TO *__restrict__ out) {
    __shared__ float tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5; // 32 x 8
    const int64_t c0 = (int64_t) blockIdx.x * 32, r0 = (int64_t) blockIdx.y * 32;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t r = r0 + ty + 8 * i, c = c0 + tx;
        float v = 0.0f;
        if (r < R && c < C) {
            const float sc = __uint_as_float((uint32_t) s[r * (C / kMxBlock) + c / kMxBlock] << 23);
            v              = __fmul_rn(fp8_to_f32<FMT>(q[r * C + c]), sc);
        }
        if constexpr (TRANSPOSE) tile[ty + 8 * i][tx] = v;
        else if (r < R && c < C) out[r * C + c] = from_f32<TO>(v);
    }
    if constexpr (TRANSPOSE) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t c = c0 + ty + 8 * i, r = r0 + tx; // out is [C][R]
            if (r < R && c < C) out[c * R + r] = from_f32<TO>(tile[tx][ty + 8 * i]);
        }
    }
}

} // namespace
} // namespace ptb

using namespace ptb;

extern "C" {
#pragma GCC visibility push(default)

int ptb_quant_mxfp8(const void *x, int x_dtype, int64_t G, int64_t M, int64_t N, void *q_row, void *s_row,
                    void *q_col, void *s_col, int row_2d_block, int col_2d_block, int q_dtype, ptb_stream_t stream) {
    PTB_REQUIRE(x_dtype == PTB_BF16 || x_dtype == PTB_F16, PTB_ERR_ARG, "MXFP8 quantise takes bf16 or fp16 input, got dtype %d", x_dtype);
    PTB_REQUIRE(is_fp8(q_dtype), PTB_ERR_ARG, "MXFP8 quantise output must be e4m3 or e5m2, got dtype %d", q_dtype);
    PTB_REQUIRE(G >= 0 && M >= 0 && N >= 0, PTB_ERR_ARG, "negative extent");
    PTB_REQUIRE(N % kMxBlock == 0, PTB_ERR_ARG, "N (%lld) must be divisible by 32", (long long) N);
    PTB_REQUIRE((q_row == nullptr) == (s_row == nullptr) && (q_col == nullptr) == (s_col == nullptr), PTB_ERR_ARG,
                "each direction needs both its data and its scale output");
    PTB_REQUIRE(q_row != nullptr || q_col != nullptr, PTB_ERR_ARG, "no output requested");
    if (G == 0 || M == 0 || N == 0) return 0;
    PTB_REQUIRE(aligned16(x) && (q_row == nullptr || aligned16(q_row)) && (q_col == nullptr || aligned16(q_col)), PTB_ERR_ARG,
                "MXFP8 quantise needs 16-byte aligned input and FP8 outputs");
    MxQuantArgs a;
    a.x = x; a.q_row = (uint8_t *) q_row; a.s_row = (uint8_t *) s_row; a.q_col = (uint8_t *) q_col; a.s_col = (uint8_t *) s_col;
    a.M = M; a.N = N; a.M_pad = cdiv<int64_t>(M, kMxPad) * kMxPad; a.N_pad = cdiv<int64_t>(N, kMxPad) * kMxPad;
    a.row_2d = row_2d_block; a.col_2d = col_2d_block;
    PTB_REQUIRE(a.M_pad / 128 <= 65535 && G <= 65535, PTB_ERR_ARG, "MXFP8 quantise: more than 65535 row tiles or groups");
    dim3 grid((unsigned) cdiv<int64_t>(a.N_pad / 128, kMxStrip), (unsigned) (a.M_pad / 128), (unsigned) G);
    cudaStream_t st = (cudaStream_t) stream;
    a.table = nullptr;
    if (x_dtype == PTB_BF16) {
        PTB_SWITCH_FP8(q_dtype, FMT, PTB_CUDA((launch_after(mx_quant_kernel<__nv_bfloat16, FMT, false>, dim3(grid), 256, 0, st, 1, a))));
    } else {
        PTB_SWITCH_FP8(q_dtype, FMT, PTB_CUDA((launch_after(mx_quant_kernel<__half, FMT, false>, dim3(grid), 256, 0, st, 1, a))));
    }
    PTB_LAUNCH_CHECK("mx_quant_kernel");
    return 0;
}

int ptb_quant_mxfp8_grouped(const void *x, int x_dtype, int64_t M, int64_t N, const int64_t *group_offs, int64_t G,
                            int64_t row_align, void *q_row, void *s_row, void *q_col, void *s_col, int64_t *row_lens_padded,
                            int64_t *row_offs_padded, int64_t *col_lens_padded, int64_t *col_offs_padded, void *block_table,
                            int row_2d_block, int col_2d_block, int q_dtype, ptb_stream_t stream) {
    PTB_REQUIRE(x_dtype == PTB_BF16 || x_dtype == PTB_F16, PTB_ERR_ARG, "MXFP8 quantise takes bf16 or fp16 input, got dtype %d", x_dtype);
    PTB_REQUIRE(is_fp8(q_dtype), PTB_ERR_ARG, "MXFP8 quantise output must be e4m3 or e5m2, got dtype %d", q_dtype);
    PTB_REQUIRE(G >= 1 && M >= 0 && N >= 0, PTB_ERR_ARG, "grouped MXFP8 quantise: at least one group, non-negative extents");
    PTB_REQUIRE(N % kMxBlock == 0, PTB_ERR_ARG, "N (%lld) must be divisible by 32", (long long) N);
    PTB_REQUIRE(row_align == 1 || row_align == 32, PTB_ERR_ARG, "row_align must be 1 or 32");
    // with no row at all (an expert-parallel rank that received nothing) x and an unpadded row copy are empty
    PTB_REQUIRE(group_offs && (M == 0 || (q_row && s_row)) && q_col && s_col && row_lens_padded && row_offs_padded &&
                    col_lens_padded && col_offs_padded && block_table,
                PTB_ERR_ARG, "grouped MXFP8 quantise: null pointer");
    PTB_REQUIRE(M < (1ll << 31), PTB_ERR_TOO_LARGE, "grouped MXFP8 quantise: too many rows");
    PTB_REQUIRE((N == 0 || aligned16(x)) && aligned16(q_row) && aligned16(q_col) && aligned16(block_table), PTB_ERR_ARG,
                "MXFP8 quantise needs 16-byte aligned input, FP8 outputs and block table");
    MxQuantArgs a;
    a.x = x ? x : q_col; // never dereferenced without rows; the zero-size copies still get a mapped address
    a.q_row = (uint8_t *) q_row; a.s_row = (uint8_t *) s_row; a.q_col = (uint8_t *) q_col; a.s_col = (uint8_t *) s_col;
    a.M = M; a.N = N;
    a.M_pad = cdiv<int64_t>(M + G * kMxPad, kMxPad) * kMxPad; // rows the column layout is allocated for (upper bound)
    a.N_pad = cdiv<int64_t>(N, kMxPad) * kMxPad;
    a.row_2d = row_2d_block; a.col_2d = col_2d_block;
    a.table  = (const int4 *) block_table;
    const int64_t nblocks = a.M_pad / kMxPad;
    PTB_REQUIRE(nblocks <= 65535, PTB_ERR_TOO_LARGE, "grouped MXFP8 quantise: more than 65535 row blocks");
    cudaStream_t st = (cudaStream_t) stream;
    PTB_CUDA((launch_after(mx_group_layout_kernel, dim3(1), 256, 0, st, 1, group_offs, G, row_align, row_lens_padded, row_offs_padded, col_lens_padded,
                                              col_offs_padded, (int4 *) block_table, nblocks)));
    PTB_LAUNCH_CHECK("mx_group_layout_kernel");
    if (N == 0) return 0;
    dim3 grid((unsigned) cdiv<int64_t>(a.N_pad / 128, kMxStrip), (unsigned) nblocks, 1);
    if (x_dtype == PTB_BF16) {
        PTB_SWITCH_FP8(q_dtype, FMT, PTB_CUDA((launch_after(mx_quant_kernel<__nv_bfloat16, FMT, true>, dim3(grid), 256, 0, st, 1, a))));
    } else {
        PTB_SWITCH_FP8(q_dtype, FMT, PTB_CUDA((launch_after(mx_quant_kernel<__half, FMT, true>, dim3(grid), 256, 0, st, 1, a))));
    }
    PTB_LAUNCH_CHECK("mx_quant_kernel");
    return 0;
}

int ptb_dequant_mxfp8(const void *q, int q_dtype, int64_t R, int64_t C, const void *scales, int transpose_out, void *out,
                      int out_dtype, ptb_stream_t stream) {
    PTB_REQUIRE(is_fp8(q_dtype) && is_hp(out_dtype), PTB_ERR_ARG, "MXFP8 dequantise: unsupported dtypes %d -> %d", q_dtype, out_dtype);
    PTB_REQUIRE(R >= 0 && C >= 0 && C % kMxBlock == 0, PTB_ERR_ARG, "MXFP8 dequantise: the inner extent (%lld) must be divisible by 32", (long long) C);
    if (R == 0 || C == 0) return 0;
    PTB_REQUIRE(cdiv<int64_t>(R, 32) <= 65535, PTB_ERR_ARG, "MXFP8 dequantise: more than 65535 row tiles");
    dim3 grid((unsigned) cdiv<int64_t>(C, 32), (unsigned) cdiv<int64_t>(R, 32));
    cudaStream_t st = (cudaStream_t) stream;
    const uint8_t *qq = (const uint8_t *) q, *ss = (const uint8_t *) scales;
#define PTB_MX_DQ(TO)                                                                                          \
    if (transpose_out) { PTB_SWITCH_FP8(q_dtype, FMT, (mx_dequant_kernel<TO, FMT, true><<<grid, 256, 0, st>>>(qq, ss, R, C, (TO *) out))); } \
    else { PTB_SWITCH_FP8(q_dtype, FMT, (mx_dequant_kernel<TO, FMT, false><<<grid, 256, 0, st>>>(qq, ss, R, C, (TO *) out))); }
    if (out_dtype == PTB_BF16) { PTB_MX_DQ(__nv_bfloat16) }
    else if (out_dtype == PTB_F16) { PTB_MX_DQ(__half) }
    else { PTB_MX_DQ(float) }
#undef PTB_MX_DQ
    PTB_LAUNCH_CHECK("mx_dequant_kernel");
    return 0;
}

#pragma GCC visibility pop
}
