// SwiGLU with routing probabilities (the activation between the gate+up and down projections of an MoE
// expert): out[t, j] = silu(x[t, j]) * x[t, H + j] * probs[t], and its backward pass.  HBM-bound
// elementwise kernels: 16-byte accesses, fp32 arithmetic, one rounding to the storage type at the end.
// The same `swiglu_prob` device function feeds the fused quantiser in ptb_quant.cu, so
// quantise(swiglu(x)) and the fused kernel produce identical bytes.
#include "ptb_common.cuh"

namespace ptb {
namespace {

// Both directions: kWarps warps per row, 8 / kWarps rows per CTA, 16 bytes per lane and access.  A row of MoE width (768
// to 2048) fills a fraction of a 256-thread CTA, and dividing a flat index by the row length costs more than the
// activation; with the warps matched to the row (at most four vectors a lane) every lane works and no index is divided.
// 32768 x 768 bf16: backward 88 -> 45 us; forward 34 -> 33 us (its division and exponential set the pace).
constexpr int kVecsPerLane = 4;

template <typename T, int kWarps>
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const T *__restrict__ x, const float *__restrict__ probs,
                                                          const int64_t *__restrict__ row_mask, int64_t rows, int64_t H,
                                                          T *__restrict__ out) {
    const int64_t r = (int64_t) blockIdx.x * (8 / kWarps) + threadIdx.x / (32 * kWarps);
    if (r >= rows) return;
    const bool live = row_mask == nullptr || row_mask[r] != 0;
    const float p   = probs[r];
    const T *xr     = x + r * 2 * H;
#pragma unroll 4
    for (int64_t c = (int64_t) (threadIdx.x % (32 * kWarps)) * 8; c < H; c += 256 * kWarps) {
        uint4 o = make_uint4(0, 0, 0, 0);
        if (live) {
            const uint4 u = *reinterpret_cast<const uint4 *>(xr + c);
            const uint4 d = *reinterpret_cast<const uint4 *>(xr + H + c);
            const T *ue = reinterpret_cast<const T *>(&u), *de = reinterpret_cast<const T *>(&d);
            T *oe = reinterpret_cast<T *>(&o);
#pragma unroll
            for (int k = 0; k < 8; ++k) oe[k] = from_f32<T>(swiglu_prob(to_f32(ue[k]), to_f32(de[k]), p));
        }
        *reinterpret_cast<uint4 *>(out + r * H + c) = o;
    }
}

// grad_x[:, :H] = g*p * down * dsilu(up), grad_x[:, H:] = g*p * silu(up),
// grad_probs = sum_j g * silu(up) * down   (primus_turbo/triton/activation/swiglu_kernel.py:196-247)
template <typename T, int kWarps>
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const T *__restrict__ grad_out, const T *__restrict__ x,
                                                          const float *__restrict__ probs,
                                                          const int64_t *__restrict__ row_mask, int64_t rows, int64_t H,
                                                          T *__restrict__ grad_x, float *__restrict__ grad_probs) {
    __shared__ float s_red[8];
    const int64_t r = (int64_t) blockIdx.x * (8 / kWarps) + threadIdx.x / (32 * kWarps);
    const bool here = r < rows; // the last CTA's spare warps still meet the barrier
    const bool live = here && (row_mask == nullptr || row_mask[r] != 0);
    const float p   = here ? probs[r] : 0.0f;
    const T *xr = x + r * 2 * H, *gr = grad_out + r * H;
    T *ur     = grad_x + r * 2 * H;
    float sum = 0.0f;
#pragma unroll 2
    for (int64_t c = (int64_t) (threadIdx.x % (32 * kWarps)) * 8; here && c < H; c += 256 * kWarps) {
        uint4 gu = make_uint4(0, 0, 0, 0), gd = make_uint4(0, 0, 0, 0);
        if (live) {
            const uint4 u = *reinterpret_cast<const uint4 *>(xr + c);
            const uint4 d = *reinterpret_cast<const uint4 *>(xr + H + c);
            const uint4 g = *reinterpret_cast<const uint4 *>(gr + c);
            const T *ue = reinterpret_cast<const T *>(&u), *de = reinterpret_cast<const T *>(&d);
            const T *ge = reinterpret_cast<const T *>(&g);
            T *gue = reinterpret_cast<T *>(&gu), *gde = reinterpret_cast<T *>(&gd);
            float part = 0.0f; // summed per vector first: the running sum stays as short as with one vector per thread
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float up = to_f32(ue[k]), down = to_f32(de[k]), go = to_f32(ge[k]);
                const float sig  = __fdiv_rn(1.0f, 1.0f + expf(-up));
                const float silu = sig * up;
                part += go * silu * down;
                const float gop = go * p;
                gde[k]          = from_f32<T>(gop * silu);
                gue[k]          = from_f32<T>(gop * (down * (sig * (1.0f + up * (1.0f - sig)))));
            }
            sum += part;
        }
        *reinterpret_cast<uint4 *>(ur + c)     = gu;
        *reinterpret_cast<uint4 *>(ur + H + c) = gd;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const int warp = threadIdx.x >> 5;
    if constexpr (kWarps == 1) {
        if (here && (threadIdx.x & 31) == 0) grad_probs[r] = sum;
    } else {
        if ((threadIdx.x & 31) == 0) s_red[warp] = sum;
        __syncthreads();
        if (here && threadIdx.x % (32 * kWarps) == 0) {
            float t = 0.0f;
#pragma unroll
            for (int k = 0; k < kWarps; ++k) t += s_red[warp + k];
            grad_probs[r] = t;
        }
    }
}

// warps that hold a row in at most kVecsPerLane vectors a lane (8 for longer rows)
#define PTB_SWITCH_ROW_WARPS(H, W, ...)                                                             \
    if ((H) <= 256 * kVecsPerLane) { constexpr int W = 1; __VA_ARGS__; }                            \
    else if ((H) <= 512 * kVecsPerLane) { constexpr int W = 2; __VA_ARGS__; }                       \
    else if ((H) <= 1024 * kVecsPerLane) { constexpr int W = 4; __VA_ARGS__; }                      \
    else { constexpr int W = 8; __VA_ARGS__; }

} // namespace
} // namespace ptb

using namespace ptb;

extern "C" {
#pragma GCC visibility push(default)

int ptb_swiglu_probs_fwd(const void *x, int dtype, const float *probs, const int64_t *row_mask, int64_t rows, int64_t H,
                         void *out, ptb_stream_t stream) {
    PTB_REQUIRE(rows >= 0 && H >= 0, PTB_ERR_ARG, "swiglu_probs_fwd: negative size");
    PTB_REQUIRE(dtype == PTB_BF16 || dtype == PTB_F16, PTB_ERR_ARG, "swiglu_probs_fwd: x must be bf16 or fp16");
    PTB_REQUIRE(H % 8 == 0, PTB_ERR_ALIGN, "swiglu_probs_fwd: the hidden size must be a multiple of 8");
    if (rows == 0 || H == 0) return 0;
    PTB_REQUIRE(x && probs && out, PTB_ERR_ARG, "swiglu_probs_fwd: null pointer");
    PTB_REQUIRE(aligned16(x) && aligned16(out), PTB_ERR_ALIGN, "swiglu_probs_fwd: buffers must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t) stream;
    PTB_SWITCH_ROW_WARPS(H, W, {
        const unsigned blocks = (unsigned) cdiv<int64_t>(rows, 8 / W);
        if (dtype == PTB_BF16)
            swiglu_fwd_kernel<__nv_bfloat16, W><<<blocks, 256, 0, st>>>((const __nv_bfloat16 *) x, probs, row_mask, rows, H, (__nv_bfloat16 *) out);
        else
            swiglu_fwd_kernel<__half, W><<<blocks, 256, 0, st>>>((const __half *) x, probs, row_mask, rows, H, (__half *) out);
    });
    PTB_LAUNCH_CHECK("swiglu_fwd_kernel");
    return 0;
}

int ptb_swiglu_probs_bwd(const void *grad_out, const void *x, int dtype, const float *probs, const int64_t *row_mask,
                         int64_t rows, int64_t H, void *grad_x, float *grad_probs, ptb_stream_t stream) {
    PTB_REQUIRE(rows >= 0 && H >= 0, PTB_ERR_ARG, "swiglu_probs_bwd: negative size");
    PTB_REQUIRE(dtype == PTB_BF16 || dtype == PTB_F16, PTB_ERR_ARG, "swiglu_probs_bwd: x must be bf16 or fp16");
    PTB_REQUIRE(H % 8 == 0, PTB_ERR_ALIGN, "swiglu_probs_bwd: the hidden size must be a multiple of 8");
    PTB_REQUIRE(rows <= 2147483647LL, PTB_ERR_TOO_LARGE, "swiglu_probs_bwd: too many rows");
    if (rows == 0) return 0;
    PTB_REQUIRE(grad_probs && probs, PTB_ERR_ARG, "swiglu_probs_bwd: null pointer");
    PTB_REQUIRE(H == 0 || (grad_out && x && grad_x), PTB_ERR_ARG, "swiglu_probs_bwd: null pointer");
    PTB_REQUIRE(aligned16(x) && aligned16(grad_out) && aligned16(grad_x), PTB_ERR_ALIGN,
                "swiglu_probs_bwd: buffers must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t) stream;
    PTB_SWITCH_ROW_WARPS(H, W, {
        const unsigned blocks = (unsigned) cdiv<int64_t>(rows, 8 / W);
        if (dtype == PTB_BF16)
            swiglu_bwd_kernel<__nv_bfloat16, W><<<blocks, 256, 0, st>>>((const __nv_bfloat16 *) grad_out, (const __nv_bfloat16 *) x, probs,
                                                                        row_mask, rows, H, (__nv_bfloat16 *) grad_x, grad_probs);
        else
            swiglu_bwd_kernel<__half, W><<<blocks, 256, 0, st>>>((const __half *) grad_out, (const __half *) x, probs, row_mask, rows, H,
                                                                 (__half *) grad_x, grad_probs);
    });
    PTB_LAUNCH_CHECK("swiglu_bwd_kernel");
    return 0;
}

#pragma GCC visibility pop
} // extern "C"
