// Row-segment copies between GPUs of one node (the expert-parallel dispatch and combine), and the
// MoE row permutation kernels that sit either side of the grouped GEMM.
//
// Dispatch and combine are the same operation: every rank holds rows that are contiguous per
// (destination rank, expert) and knows, from the routing counts of all ranks, the row at which each
// such segment starts in the destination's buffer.  One kernel copies all segments of a rank with plain
// 16-byte loads from local memory and plain 16-byte stores to the destination -- peer memory mapped
// into this process (NVLink / NVSwitch) or local memory for the rank's own share -- so rows land in
// expert-major order, ready for the grouped GEMM, with no staging pass on either side.  The copy kernel
// waits on nothing.  Ordering between ranks: either a collective afterwards, or the copy's own signal --
// the last CTA to finish stores the exchange's sequence number into a slot of every destination's flag
// array (release, system scope, after every thread has fenced its data stores), and the destination runs
// a one-warp kernel that waits, with a time limit, until all sources' slots carry that number.
#include "ptb_common.cuh"

namespace ptb {
namespace {

constexpr int kMaxPeers    = 16;
constexpr int kCopyThreads = 512;
constexpr int kChunkBytes  = 4 * kCopyThreads * 16; // 32 KiB per work item: four 16-byte loads in flight per thread
constexpr int kMaxSegments = 8192;

struct CopyArgs {
    const uint8_t *src;
    uint8_t *dst[kMaxPeers];
    const int64_t *segs; // [nseg][4]: first source row, first destination row, rows, destination rank
    int nseg;
    int n_ranks;
    int64_t row_bytes;
    // optional arrival signal (done == nullptr: none)
    uint32_t *flag[kMaxPeers]; // per destination rank: this rank's slot in that rank's flag array
    uint32_t *done;            // local counter of finished CTAs, zero between launches
    uint32_t seq;
};

constexpr uint64_t kFlagWaitLimitNs = 20000000000ull; // 20 s: ranks of one job are never this far apart

__device__ __forceinline__ void st_release_sys(uint32_t *p, uint32_t v) {
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// set to 1 by a copy whose segment table names a rank outside [0, n_ranks) (that segment is skipped),
// to 2 by a flag wait that ran out of time
__device__ int g_copy_error = 0;

__global__ void __launch_bounds__(kCopyThreads) copy_segments_kernel(const CopyArgs a) {
    // chunk-count prefix over the segments, built by the whole CTA (nseg <= kMaxSegments)
    __shared__ int s_prefix[kMaxSegments + 1];
    __shared__ int s_warp[kCopyThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int run = 0;
    for (int base = 0; base < a.nseg; base += kCopyThreads) {
        const int s = base + tid;
        int cnt     = 0;
        if (s < a.nseg) cnt = (int) ((a.segs[4 * s + 2] * a.row_bytes + kChunkBytes - 1) / kChunkBytes);
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += n;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        int before = run;
        for (int w = 0; w < warp; ++w) before += s_warp[w];
        if (s < a.nseg) s_prefix[s + 1] = before + inc;
        int total = 0;
        for (int w = 0; w < kCopyThreads / 32; ++w) total += s_warp[w];
        run += total;
        __syncthreads();
    }
    if (tid == 0) s_prefix[0] = 0;
    __syncthreads();
    const int total_chunks = s_prefix[a.nseg];

    for (int c = blockIdx.x; c < total_chunks; c += gridDim.x) {
        // segment that holds chunk c: last s with prefix[s] <= c
        int lo = 0, hi = a.nseg - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_prefix[mid] <= c) lo = mid;
            else hi = mid - 1;
        }
        const int64_t *sg = a.segs + 4 * lo;
        const int64_t rank = sg[3];
        if (rank < 0 || rank >= a.n_ranks) {
            if (tid == 0) atomicExch(&g_copy_error, 1);
            continue;
        }
        const int64_t seg_bytes = sg[2] * a.row_bytes;
        const int64_t off       = (int64_t) (c - s_prefix[lo]) * kChunkBytes;
        const int64_t n         = min((int64_t) kChunkBytes, seg_bytes - off);
        const uint4 *src = reinterpret_cast<const uint4 *>(a.src + sg[0] * a.row_bytes + off);
        uint4 *dst       = reinterpret_cast<uint4 *>(a.dst[rank] + sg[1] * a.row_bytes + off);
        const int nvec   = (int) (n >> 4);
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = tid + i * kCopyThreads;
            if (j < nvec) v[i] = __ldg(src + j);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = tid + i * kCopyThreads;
            if (j < nvec) dst[j] = v[i];
        }
    }
    if (a.done != nullptr) {
        __threadfence_system(); // this thread's stores, wherever they went, before the CTA counts itself
        __syncthreads();
        if (tid == 0) {
            __threadfence_system();
            if (atomicAdd(a.done, 1u) == gridDim.x - 1) {
                __threadfence_system();
                for (int r = 0; r < a.n_ranks; ++r) st_release_sys(a.flag[r], a.seq);
                *a.done = 0; // the next launch on this stream starts after this kernel has ended
            }
        }
    }
}

// One warp: lane r waits until flags[r] has reached `seq` (sequence numbers only grow; the comparison
// survives wrap-around).  On expiry it records the failure and returns -- the stream goes on with
// whatever arrived, and the host finds the status word set.
__global__ void __launch_bounds__(32) wait_flags_kernel(const uint32_t *flags, int n, uint32_t seq) {
    const int r = threadIdx.x;
    if (r >= n) return;
    uint64_t t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    while ((int32_t) (ld_acquire_sys(flags + r) - seq) < 0) {
        __nanosleep(100);
        uint64_t t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > kFlagWaitLimitNs) {
            atomicExch(&g_copy_error, 2);
            break;
        }
    }
}

// ---- row permutation: out[i] = in[index[i]] (gather) for rows of `row_bytes` bytes -------------------
// One warp per row, 16-byte accesses; rows whose index is negative are written as zeros (dropped tokens).
__global__ void __launch_bounds__(256) gather_rows_kernel(const uint8_t *__restrict__ in, const int64_t *__restrict__ index,
                                                           int64_t n_out, int64_t n_in, int64_t row_bytes,
                                                           uint8_t *__restrict__ out) {
    const int lane  = threadIdx.x & 31;
    const int64_t w = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t) gridDim.x * blockDim.x) >> 5;
    const int64_t nvec = row_bytes >> 4;
    for (int64_t r = w; r < n_out; r += nw) {
        const int64_t s = index[r];
        uint4 *dst      = reinterpret_cast<uint4 *>(out + r * row_bytes);
        if (s < 0 || s >= n_in) {
            for (int64_t j = lane; j < nvec; j += 32) dst[j] = make_uint4(0, 0, 0, 0);
        } else {
            const uint4 *src = reinterpret_cast<const uint4 *>(in + s * row_bytes);
            for (int64_t j = lane; j < nvec; j += 32) dst[j] = __ldg(src + j);
        }
    }
}

// ---- MoE token permutation: routing map -> expert-major positions --------------------------------------
// routing_map [T, E] (one byte per entry, non-zero = token t goes to expert e).  Position of (t, e) in
// the permuted order = rows of experts below e + tokens below t routed to e: a stable counting sort in
// three passes over blocks of kTokBlock tokens (count per block and expert, scan, assign).
//
// Bound by latency: the map is a byte an entry, so a thread that walks an expert's 256 tokens one dependent byte load
// after another took 50 us a pass.  A tile of 256 tokens x 64 experts is turned into bit masks instead (one thread per
// token, 16 bytes a load, one ballot per expert and warp); counts and positions are popcounts of those.  4096 x 64, two
// calls: count 100 -> 6 us, assign 47 -> 16 us.
constexpr int kTokBlock = 256, kExpTile = 64, kTokWarps = kTokBlock / 32;

// s_mask[w][e]: bit i = token 32 w + i of the block is routed to expert e0 + e
__device__ __forceinline__ void moe_tile_masks(const uint8_t *__restrict__ map, int64_t T, int64_t E, int64_t t0, int64_t e0,
                                               uint32_t (&s_mask)[kTokWarps][kExpTile]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t t    = t0 + threadIdx.x;
    const uint8_t *row = map + t * E + e0;
    const bool vec     = E % 16 == 0 && (reinterpret_cast<uintptr_t>(map) & 15u) == 0;
#pragma unroll 1
    for (int h = 0; h < kExpTile; h += 32) {
        uint32_t mine = 0;
#pragma unroll
        for (int c = 0; c < 32; c += 16) {
            uint4 raw  = make_uint4(0, 0, 0, 0);
            uint8_t *r = reinterpret_cast<uint8_t *>(&raw);
            if (t < T) {
                if (vec) {
                    if (e0 + h + c < E) raw = *reinterpret_cast<const uint4 *>(row + h + c);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = e0 + h + c + j < E ? row[h + c + j] : (uint8_t) 0;
                }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const uint32_t m = __ballot_sync(0xffffffffu, r[j] != 0);
                if (lane == c + j) mine = m;
            }
        }
        s_mask[w][h + lane] = mine;
    }
    __syncthreads();
}

// grid: (token blocks, expert tiles)
__global__ void __launch_bounds__(kTokBlock) moe_count_kernel(const uint8_t *__restrict__ map, int64_t T, int64_t E,
                                                              int *__restrict__ block_counts) {
    __shared__ uint32_t s_mask[kTokWarps][kExpTile];
    const int64_t e0 = (int64_t) blockIdx.y * kExpTile, e = e0 + threadIdx.x;
    moe_tile_masks(map, T, E, (int64_t) blockIdx.x * kTokBlock, e0, s_mask);
    if (threadIdx.x < kExpTile && e < E) {
        int c = 0;
#pragma unroll
        for (int w = 0; w < kTokWarps; ++w) c += __popc(s_mask[w][threadIdx.x]);
        block_counts[(int64_t) blockIdx.x * E + e] = c;
    }
}

// one CTA: per expert, exclusive scan of the block counts over the token blocks (eight loads at a time: they do not
// depend on the running sum); then the experts' first positions, an exclusive scan over experts
__global__ void __launch_bounds__(256) moe_scan_kernel(int *__restrict__ block_counts, int64_t B, int64_t E,
                                                        int64_t *__restrict__ tokens_per_expert,
                                                        int64_t *__restrict__ expert_start) {
    __shared__ int64_t s_cnt[1024], s_scan[256]; // at most kMaxExperts experts (checked by the launcher)
    const int tid = threadIdx.x;
    for (int64_t e = tid; e < E; e += blockDim.x) {
        int run = 0;
        for (int64_t b0 = 0; b0 < B; b0 += 8) {
            int c[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) c[u] = b0 + u < B ? block_counts[(b0 + u) * E + e] : 0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (b0 + u < B) block_counts[(b0 + u) * E + e] = run;
                run += c[u];
            }
        }
        tokens_per_expert[e] = run;
        s_cnt[e]             = run;
    }
    __syncthreads();
    const int64_t per = cdiv<int64_t>(E, 256), g0 = imin(tid * per, E), g1 = imin(g0 + per, E);
    int64_t local = 0;
    for (int64_t e = g0; e < g1; ++e) local += s_cnt[e];
    s_scan[tid] = local;
    __syncthreads();
    for (int off = 1; off < 256; off <<= 1) {
        const int64_t add = (tid >= off) ? s_scan[tid - off] : 0;
        __syncthreads();
        s_scan[tid] += add;
        __syncthreads();
    }
    int64_t run = s_scan[tid] - local;
    for (int64_t e = g0; e < g1; ++e) {
        expert_start[e] = run;
        run += s_cnt[e];
    }
    if (tid == 255) expert_start[E] = s_scan[255];
}

// positions fit 32 bits: the launcher requires T * E < 2^31
__global__ void __launch_bounds__(kTokBlock) moe_assign_kernel(const uint8_t *__restrict__ map, int64_t T, int64_t E,
                                                               const int *__restrict__ block_counts,
                                                               const int64_t *__restrict__ expert_start, int64_t capacity,
                                                               int *__restrict__ row_id_map,
                                                               int64_t *__restrict__ sorted_indices) {
    __shared__ uint32_t s_mask[kTokWarps][kExpTile];
    __shared__ int s_base[kTokWarps][kExpTile]; // position of the first token of each 32 that goes to the expert
    const int64_t t0 = (int64_t) blockIdx.x * kTokBlock, e0 = (int64_t) blockIdx.y * kExpTile;
    moe_tile_masks(map, T, E, t0, e0, s_mask);
    if (threadIdx.x < kExpTile && e0 + threadIdx.x < E) {
        int pos = (int) expert_start[e0 + threadIdx.x] + block_counts[(int64_t) blockIdx.x * E + e0 + threadIdx.x];
#pragma unroll
        for (int w = 0; w < kTokWarps; ++w) {
            s_base[w][threadIdx.x] = pos;
            pos += __popc(s_mask[w][threadIdx.x]);
        }
    }
    __syncthreads();
    const int e = threadIdx.x % kExpTile;
    if (e0 + e >= E) return;
    for (int tl = threadIdx.x / kExpTile; tl < kTokBlock && t0 + tl < T; tl += kTokBlock / kExpTile) {
        const uint32_t m = s_mask[tl >> 5][e], bit = 1u << (tl & 31);
        const int pos = s_base[tl >> 5][e] + __popc(m & (bit - 1));
        const bool ok = (m & bit) != 0 && pos < capacity;
        row_id_map[(t0 + tl) * E + e0 + e] = ok ? pos : -1;
        if (ok && sorted_indices != nullptr) sorted_indices[pos] = t0 + tl;
    }
}

// ---- routing probabilities between the [T, E] table and one value per permuted row -------------------------
// V is an unsigned integer of the element's size: values are moved, not computed with.
template <typename V>
__global__ void __launch_bounds__(256) moe_probs_to_rows_kernel(const int *__restrict__ row_id_map, const V *__restrict__ probs,
                                                                int64_t n, V *__restrict__ rows) {
    for (int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x) {
        const int id = row_id_map[i];
        if (id >= 0) rows[id] = probs[i];
    }
}
template <typename V>
__global__ void __launch_bounds__(256) moe_rows_to_probs_kernel(const int *__restrict__ row_id_map, const V *__restrict__ rows,
                                                                int64_t n, V *__restrict__ probs) {
    for (int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x) {
        const int id = row_id_map[i];
        probs[i]     = id >= 0 ? rows[id] : (V) 0;
    }
}

// zeros rows [sum(counts), n_rows): the rows of a permuted buffer that no (token, expert) pair owns
__global__ void __launch_bounds__(256) zero_rows_after_kernel(const int64_t *__restrict__ counts, int64_t G, int64_t n_rows,
                                                              int64_t row_bytes, uint8_t *__restrict__ out) {
    __shared__ int64_t s_sum[256];
    int64_t sum = 0;
    for (int64_t g = threadIdx.x; g < G; g += 256) sum += counts[g];
    s_sum[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) s_sum[threadIdx.x] += s_sum[threadIdx.x + o];
        __syncthreads();
    }
    const int64_t from = imin(s_sum[0], n_rows) * row_bytes, end = n_rows * row_bytes;
    const int64_t tid = (int64_t) blockIdx.x * 256 + threadIdx.x, step = (int64_t) gridDim.x * 256;
    if (row_bytes % 16 == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
        for (int64_t i = from / 16 + tid; i < end / 16; i += step) reinterpret_cast<uint4 *>(out)[i] = make_uint4(0, 0, 0, 0);
    } else {
        for (int64_t i = from + tid; i < end; i += step) out[i] = 0;
    }
}

// ---- weighted row gather: out[i] = cast(float(in[index[i]]) * w[i]) ---------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) gather_rows_scaled_kernel(const T *__restrict__ in, const int64_t *__restrict__ index,
                                                                  const float *__restrict__ weights, int64_t n_out,
                                                                  int64_t n_in, int64_t H, T *__restrict__ out) {
    const int lane   = threadIdx.x & 31;
    const int64_t w  = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t) gridDim.x * blockDim.x) >> 5;
    for (int64_t r = w; r < n_out; r += nw) {
        const int64_t s = index[r];
        const float wt  = weights[r];
        const bool ok   = s >= 0 && s < n_in;
        for (int64_t j = lane; j < H; j += 32)
            out[r * H + j] = from_f32<T>(ok ? __fmul_rn(to_f32(in[s * H + j]), wt) : 0.0f);
    }
}

// ---- un-permute: out[t] = sum over the experts e of token t, in increasing e, of in[pos(t,e)] * p(t,e) ------
// One warp per token.  The (at most E) positions of the token are compacted into shared memory first,
// then every lane walks its columns once per position.  Products and sums are separate fp32 operations
// (no contraction), accumulated in expert order: the result equals a sequential fp32 scatter-add.
constexpr int kUnpermWarps = 4;
constexpr int kMaxExperts  = 1024;

template <typename T, bool WITH_GRAD>
__global__ void __launch_bounds__(kUnpermWarps * 32) unpermute_kernel(
    const T *__restrict__ in, const int *__restrict__ row_id_map, const float *__restrict__ probs, int64_t T_, int64_t E,
    int64_t H, T *__restrict__ out,
    // WITH_GRAD: `in` is the gradient of the un-permuted rows [T, H], `fwd_in` the permuted rows of the
    // forward pass; writes grad_in[pos] = g[t] * p and grad_probs[t, e] = dot(g[t], fwd_in[pos])
    const T *__restrict__ fwd_in, float *__restrict__ grad_probs) {
    __shared__ int s_pos[kUnpermWarps][kMaxExperts];
    __shared__ int s_exp[kUnpermWarps][kMaxExperts];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t = (int64_t) blockIdx.x * kUnpermWarps + warp;
    if (t >= T_) return;
    int n = 0;
    for (int64_t base = 0; base < E; base += 32) {
        const int64_t e = base + lane;
        const int id    = e < E ? row_id_map[t * E + e] : -1;
        const unsigned m = __ballot_sync(0xffffffffu, id >= 0);
        if (id >= 0) {
            const int k  = n + __popc(m & ((1u << lane) - 1));
            s_pos[warp][k] = id;
            s_exp[warp][k] = (int) e;
        }
        if (WITH_GRAD && grad_probs != nullptr && e < E && id < 0) grad_probs[t * E + e] = 0.0f;
        n += __popc(m);
    }
    __syncwarp();
    if constexpr (!WITH_GRAD) {
        for (int64_t j = lane; j < H; j += 32) {
            float acc = 0.0f;
            for (int k = 0; k < n; ++k) {
                float v = to_f32(in[(int64_t) s_pos[warp][k] * H + j]);
                if (probs != nullptr) v = __fmul_rn(v, probs[t * E + s_exp[warp][k]]);
                acc = __fadd_rn(acc, v);
            }
            out[t * H + j] = from_f32<T>(acc);
        }
    } else {
        for (int k = 0; k < n; ++k) {
            const int64_t pos = s_pos[warp][k];
            const float p     = probs != nullptr ? probs[t * E + s_exp[warp][k]] : 1.0f;
            float dot         = 0.0f;
            for (int64_t j = lane; j < H; j += 32) {
                const float g = to_f32(in[t * H + j]);
                out[pos * H + j] = from_f32<T>(__fmul_rn(g, p));
                if (grad_probs != nullptr) dot += g * to_f32(fwd_in[pos * H + j]);
            }
            if (grad_probs != nullptr) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
                if (lane == 0) grad_probs[t * E + s_exp[warp][k]] = dot;
            }
        }
    }
}

// The same for rows of whole, aligned 16-byte vectors, bound by HBM (every permuted row is read or written once).  A warp
// takes one token and a slice of kUnpermVecs vectors per lane; four copies of the token are in flight at a time and are
// added in expert order, each column by one lane, so the values are those of the element form.  The element form moved 64
// bytes per warp and load: 4096 tokens x 8 copies x 2048 bf16, both merges of a layer, took 184 us, this takes
// 64; gradients 41 -> 25 us.  With grad_probs one warp has to see the whole row (one slice).
constexpr int kUnpermVecs = 2, kUnpermCopies = 4;

template <typename T, bool WITH_GRAD>
__global__ void __launch_bounds__(kUnpermWarps * 32) unpermute_vec_kernel(
    const T *__restrict__ in, const int *__restrict__ row_id_map, const float *__restrict__ probs, int64_t T_, int64_t E,
    int64_t H, T *__restrict__ out, const T *__restrict__ fwd_in, float *__restrict__ grad_probs) {
    extern __shared__ int s_list[]; // per warp: E positions, E experts
    constexpr int V = 16 / sizeof(T);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t = (int64_t) blockIdx.x * kUnpermWarps + warp;
    if (t >= T_) return;
    int *s_pos = s_list + warp * 2 * E, *s_exp = s_pos + E;
    int n = 0;
    for (int64_t base = 0; base < E; base += 32) {
        const int64_t e  = base + lane;
        const int id     = e < E ? row_id_map[t * E + e] : -1;
        const unsigned m = __ballot_sync(0xffffffffu, id >= 0);
        if (id >= 0) {
            const int k = n + __popc(m & ((1u << lane) - 1));
            s_pos[k]    = id;
            s_exp[k]    = (int) e;
        }
        if (WITH_GRAD && grad_probs != nullptr && e < E && id < 0) grad_probs[t * E + e] = 0.0f;
        n += __popc(m);
    }
    __syncwarp();
    const int64_t col0 = ((int64_t) blockIdx.y * kUnpermVecs * 32 + lane) * V; // vector v of a lane: col0 + 32 * V * v
    if constexpr (!WITH_GRAD) {
        float acc[kUnpermVecs][V];
#pragma unroll
        for (int v = 0; v < kUnpermVecs; ++v)
#pragma unroll
            for (int j = 0; j < V; ++j) acc[v][j] = 0.0f;
        for (int k = 0; k < n; k += kUnpermCopies) {
            uint4 raw[kUnpermCopies][kUnpermVecs];
            float p[kUnpermCopies];
#pragma unroll
            for (int u = 0; u < kUnpermCopies; ++u) {
                if (k + u >= n) continue;
                p[u] = probs != nullptr ? probs[t * E + s_exp[k + u]] : 1.0f;
#pragma unroll
                for (int v = 0; v < kUnpermVecs; ++v) {
                    const int64_t c = col0 + 32 * V * v;
                    if (c < H) raw[u][v] = *reinterpret_cast<const uint4 *>(in + (int64_t) s_pos[k + u] * H + c);
                }
            }
#pragma unroll
            for (int u = 0; u < kUnpermCopies; ++u) {
                if (k + u >= n) continue;
#pragma unroll
                for (int v = 0; v < kUnpermVecs; ++v) {
                    const T *e = reinterpret_cast<const T *>(&raw[u][v]);
#pragma unroll
                    for (int j = 0; j < V; ++j) {
                        float x = to_f32(e[j]);
                        if (probs != nullptr) x = __fmul_rn(x, p[u]);
                        acc[v][j] = __fadd_rn(acc[v][j], x);
                    }
                }
            }
        }
#pragma unroll
        for (int v = 0; v < kUnpermVecs; ++v) {
            const int64_t c = col0 + 32 * V * v;
            if (c >= H) continue;
            uint4 o;
#pragma unroll
            for (int j = 0; j < V; ++j) reinterpret_cast<T *>(&o)[j] = from_f32<T>(acc[v][j]);
            *reinterpret_cast<uint4 *>(out + t * H + c) = o;
        }
    } else if (grad_probs == nullptr) {
#pragma unroll
        for (int v = 0; v < kUnpermVecs; ++v) {
            const int64_t c = col0 + 32 * V * v;
            if (c >= H) continue;
            const uint4 g = *reinterpret_cast<const uint4 *>(in + t * H + c);
            for (int k = 0; k < n; ++k) {
                uint4 o = g;
                if (probs != nullptr) {
                    const float p = probs[t * E + s_exp[k]];
#pragma unroll
                    for (int j = 0; j < V; ++j)
                        reinterpret_cast<T *>(&o)[j] = from_f32<T>(__fmul_rn(to_f32(reinterpret_cast<const T *>(&g)[j]), p));
                }
                *reinterpret_cast<uint4 *>(out + (int64_t) s_pos[k] * H + c) = o;
            }
        }
    } else {
        for (int k = 0; k < n; ++k) {
            const int64_t pos = s_pos[k];
            const float p     = probs != nullptr ? probs[t * E + s_exp[k]] : 1.0f;
            float dot         = 0.0f;
#pragma unroll 4
            for (int64_t c = lane * V; c < H; c += 32 * V) {
                const uint4 g = *reinterpret_cast<const uint4 *>(in + t * H + c);
                const uint4 f = *reinterpret_cast<const uint4 *>(fwd_in + pos * H + c);
                uint4 o;
                float part = 0.0f; // summed per vector first: the running sum has no more terms than the element form's
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    const float gv = to_f32(reinterpret_cast<const T *>(&g)[j]);
                    reinterpret_cast<T *>(&o)[j] = from_f32<T>(__fmul_rn(gv, p));
                    part += gv * to_f32(reinterpret_cast<const T *>(&f)[j]);
                }
                dot += part;
                *reinterpret_cast<uint4 *>(out + pos * H + c) = o;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            if (lane == 0) grad_probs[t * E + s_exp[k]] = dot;
        }
    }
}

// whole 16-byte vectors per row, every buffer on a 16-byte boundary, and at most 65535 slices
template <typename T> bool unpermute_vec_ok(const void *a, const void *b, const void *c, int64_t H) {
    return H % (16 / (int64_t) sizeof(T)) == 0 && H <= 65535LL * 256 && aligned16(a) && aligned16(b) && (c == nullptr || aligned16(c));
}
template <typename T> unsigned unpermute_slices(int64_t H) {
    return (unsigned) cdiv<int64_t>(H, (int64_t) kUnpermVecs * 32 * (16 / (int64_t) sizeof(T)));
}

} // namespace
} // namespace ptb

using namespace ptb;

extern "C" {
#pragma GCC visibility push(default)

static int copy_segments_impl(const void *src_base, void *const *dst_bases, int n_ranks, const int64_t *segments,
                              int64_t nseg, int64_t row_bytes, int num_ctas, void *const *flag_slots, void *done_counter,
                              uint32_t seq, ptb_stream_t stream);

int ptb_copy_segments(const void *src_base, void *const *dst_bases, int n_ranks, const int64_t *segments, int64_t nseg,
                      int64_t row_bytes, int num_ctas, ptb_stream_t stream) {
    return copy_segments_impl(src_base, dst_bases, n_ranks, segments, nseg, row_bytes, num_ctas, nullptr, nullptr, 0, stream);
}

int ptb_copy_segments_signal(const void *src_base, void *const *dst_bases, int n_ranks, const int64_t *segments,
                             int64_t nseg, int64_t row_bytes, int num_ctas, void *const *flag_slots, void *done_counter,
                             uint32_t seq, ptb_stream_t stream) {
    PTB_REQUIRE(flag_slots && done_counter, PTB_ERR_ARG, "copy_segments_signal: null flag slots or counter");
    return copy_segments_impl(src_base, dst_bases, n_ranks, segments, nseg, row_bytes, num_ctas, flag_slots, done_counter, seq,
                              stream);
}

int ptb_wait_flags(const void *flags, int n, uint32_t seq, ptb_stream_t stream) {
    PTB_REQUIRE(flags && n >= 1 && n <= 32, PTB_ERR_ARG, "wait_flags: 1 to 32 flags");
    wait_flags_kernel<<<1, 32, 0, (cudaStream_t) stream>>>((const uint32_t *) flags, n, seq);
    PTB_LAUNCH_CHECK("wait_flags_kernel");
    return 0;
}

static int copy_segments_impl(const void *src_base, void *const *dst_bases, int n_ranks, const int64_t *segments,
                              int64_t nseg, int64_t row_bytes, int num_ctas, void *const *flag_slots, void *done_counter,
                              uint32_t seq, ptb_stream_t stream) {
    PTB_REQUIRE(n_ranks >= 1 && n_ranks <= kMaxPeers, PTB_ERR_TOO_LARGE, "copy_segments: 1 to %d ranks, got %d", kMaxPeers,
                n_ranks);
    PTB_REQUIRE(nseg >= 0 && nseg <= kMaxSegments, PTB_ERR_TOO_LARGE, "copy_segments: at most %d segments", kMaxSegments);
    PTB_REQUIRE(row_bytes > 0 && row_bytes % 16 == 0, PTB_ERR_ALIGN, "copy_segments: row size %lld is not a multiple of 16 bytes",
                (long long) row_bytes);
    if (nseg == 0 && flag_slots == nullptr) return 0;
    PTB_REQUIRE(dst_bases && (nseg == 0 || (src_base && segments)), PTB_ERR_ARG, "copy_segments: null pointer");
    PTB_REQUIRE(aligned16(src_base), PTB_ERR_ALIGN, "copy_segments: source is not 16-byte aligned");
    CopyArgs a{};
    a.src = (const uint8_t *) src_base;
    for (int r = 0; r < n_ranks; ++r) {
        PTB_REQUIRE(dst_bases[r] && aligned16(dst_bases[r]), PTB_ERR_ALIGN,
                    "copy_segments: destination of rank %d is null or not 16-byte aligned", r);
        a.dst[r] = (uint8_t *) dst_bases[r];
    }
    a.segs = segments; a.nseg = (int) nseg; a.n_ranks = n_ranks; a.row_bytes = row_bytes;
    if (flag_slots != nullptr) {
        for (int r = 0; r < n_ranks; ++r) {
            PTB_REQUIRE(flag_slots[r] && (reinterpret_cast<uintptr_t>(flag_slots[r]) & 3u) == 0, PTB_ERR_ALIGN,
                        "copy_segments_signal: flag slot of rank %d is null or misaligned", r);
            a.flag[r] = (uint32_t *) flag_slots[r];
        }
        a.done = (uint32_t *) done_counter;
        a.seq  = seq;
    }
    int dev = 0, sms = 0;
    PTB_CUDA(cudaGetDevice(&dev));
    PTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int grid = (num_ctas > 0) ? num_ctas : sms;
    copy_segments_kernel<<<grid, kCopyThreads, 0, (cudaStream_t) stream>>>(a);
    PTB_LAUNCH_CHECK("copy_segments_kernel");
    return 0;
}

int ptb_enable_peer_access(int peer_device) {
    int dev = -1;
    PTB_CUDA(cudaGetDevice(&dev));
    if (peer_device == dev) return 0;
    int can = 0;
    PTB_CUDA(cudaDeviceCanAccessPeer(&can, dev, peer_device));
    PTB_REQUIRE(can, PTB_ERR_UNSUPPORTED, "device %d cannot address the memory of device %d", dev, peer_device);
    const cudaError_t e = cudaDeviceEnablePeerAccess(peer_device, 0);
    if (e == cudaErrorPeerAccessAlreadyEnabled) {
        (void) cudaGetLastError(); // not an error: clear it
        return 0;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceEnablePeerAccess");
    return 0;
}

int ptb_copy_segments_status(int *status, int reset) {
    PTB_REQUIRE(status, PTB_ERR_ARG, "copy_segments_status: null pointer");
    PTB_CUDA(cudaMemcpyFromSymbol(status, g_copy_error, sizeof(int)));
    if (reset) {
        int zero = 0;
        PTB_CUDA(cudaMemcpyToSymbol(g_copy_error, &zero, sizeof(int)));
    }
    return 0;
}

int ptb_gather_rows(const void *in, const int64_t *index, int64_t n_out, int64_t n_in, int64_t row_bytes, void *out,
                    ptb_stream_t stream) {
    PTB_REQUIRE(n_out >= 0 && n_in >= 0, PTB_ERR_ARG, "gather_rows: negative size");
    PTB_REQUIRE(row_bytes > 0 && row_bytes % 16 == 0, PTB_ERR_ALIGN, "gather_rows: row size %lld is not a multiple of 16 bytes",
                (long long) row_bytes);
    if (n_out == 0) return 0;
    PTB_REQUIRE(index && out && (n_in == 0 || in), PTB_ERR_ARG, "gather_rows: null pointer");
    PTB_REQUIRE(aligned16(out) && (n_in == 0 || aligned16(in)), PTB_ERR_ALIGN, "gather_rows: buffers must be 16-byte aligned");
    const int64_t warps = n_out;
    const int blocks    = (int) imin(cdiv<int64_t>(warps, 8), 148 * 16);
    gather_rows_kernel<<<blocks, 256, 0, (cudaStream_t) stream>>>((const uint8_t *) in, index, n_out, n_in, row_bytes,
                                                                   (uint8_t *) out);
    PTB_LAUNCH_CHECK("gather_rows_kernel");
    return 0;
}

int ptb_moe_row_id_map(const void *routing_map, int64_t T, int64_t E, int64_t capacity, int32_t *row_id_map,
                       int64_t *tokens_per_expert, int64_t *sorted_indices, void *workspace, ptb_stream_t stream) {
    PTB_REQUIRE(T >= 0 && E >= 0 && capacity >= 0, PTB_ERR_ARG, "moe_row_id_map: negative size");
    PTB_REQUIRE(E <= kMaxExperts, PTB_ERR_TOO_LARGE, "moe_row_id_map: at most %d experts", kMaxExperts);
    PTB_REQUIRE(T * E < 2147483647LL && capacity < 2147483647LL, PTB_ERR_TOO_LARGE, "moe_row_id_map: problem too large");
    if (E == 0) return 0;
    PTB_REQUIRE(tokens_per_expert && workspace, PTB_ERR_ARG, "moe_row_id_map: null pointer");
    const int64_t B = cdiv<int64_t>(T, kTokBlock);
    int *block_counts     = (int *) workspace;                               // [B, E] int32
    int64_t *expert_start = (int64_t *) ((uint8_t *) workspace + ((B * E * 4 + 15) / 16) * 16); // [E + 1] int64
    cudaStream_t st = (cudaStream_t) stream;
    const dim3 grid((unsigned) B, (unsigned) cdiv<int64_t>(E, kExpTile));
    if (T > 0) {
        PTB_REQUIRE(routing_map && row_id_map, PTB_ERR_ARG, "moe_row_id_map: null pointer");
        moe_count_kernel<<<grid, kTokBlock, 0, st>>>((const uint8_t *) routing_map, T, E, block_counts);
        PTB_LAUNCH_CHECK("moe_count_kernel");
    }
    moe_scan_kernel<<<1, 256, 0, st>>>(block_counts, B, E, tokens_per_expert, expert_start);
    PTB_LAUNCH_CHECK("moe_scan_kernel");
    if (T > 0) {
        moe_assign_kernel<<<grid, kTokBlock, 0, st>>>((const uint8_t *) routing_map, T, E, block_counts, expert_start,
                                                         capacity, row_id_map, sorted_indices);
        PTB_LAUNCH_CHECK("moe_assign_kernel");
    }
    return 0;
}

int ptb_moe_probs_to_rows(const int32_t *row_id_map, const void *probs, int elem_bytes, int64_t n, void *rows, ptb_stream_t stream) {
    PTB_REQUIRE(n >= 0, PTB_ERR_ARG, "moe_probs_to_rows: negative size");
    if (n == 0) return 0;
    PTB_REQUIRE(row_id_map && probs && rows, PTB_ERR_ARG, "moe_probs_to_rows: null pointer");
    const int blocks = (int) imin(cdiv<int64_t>(n, 256), 148 * 8);
    cudaStream_t st  = (cudaStream_t) stream;
    switch (elem_bytes) {
    case 1: moe_probs_to_rows_kernel<uint8_t><<<blocks, 256, 0, st>>>(row_id_map, (const uint8_t *) probs, n, (uint8_t *) rows); break;
    case 2: moe_probs_to_rows_kernel<uint16_t><<<blocks, 256, 0, st>>>(row_id_map, (const uint16_t *) probs, n, (uint16_t *) rows); break;
    case 4: moe_probs_to_rows_kernel<uint32_t><<<blocks, 256, 0, st>>>(row_id_map, (const uint32_t *) probs, n, (uint32_t *) rows); break;
    case 8: moe_probs_to_rows_kernel<uint64_t><<<blocks, 256, 0, st>>>(row_id_map, (const uint64_t *) probs, n, (uint64_t *) rows); break;
    default: return fail(PTB_ERR_ARG, "moe_probs_to_rows: element size %d", elem_bytes);
    }
    PTB_LAUNCH_CHECK("moe_probs_to_rows_kernel");
    return 0;
}

int ptb_moe_rows_to_probs(const int32_t *row_id_map, const void *rows, int elem_bytes, int64_t n, void *probs, ptb_stream_t stream) {
    PTB_REQUIRE(n >= 0, PTB_ERR_ARG, "moe_rows_to_probs: negative size");
    if (n == 0) return 0;
    PTB_REQUIRE(row_id_map && probs, PTB_ERR_ARG, "moe_rows_to_probs: null pointer"); // no rows: the map names none
    const int blocks = (int) imin(cdiv<int64_t>(n, 256), 148 * 8);
    cudaStream_t st  = (cudaStream_t) stream;
    switch (elem_bytes) {
    case 1: moe_rows_to_probs_kernel<uint8_t><<<blocks, 256, 0, st>>>(row_id_map, (const uint8_t *) rows, n, (uint8_t *) probs); break;
    case 2: moe_rows_to_probs_kernel<uint16_t><<<blocks, 256, 0, st>>>(row_id_map, (const uint16_t *) rows, n, (uint16_t *) probs); break;
    case 4: moe_rows_to_probs_kernel<uint32_t><<<blocks, 256, 0, st>>>(row_id_map, (const uint32_t *) rows, n, (uint32_t *) probs); break;
    case 8: moe_rows_to_probs_kernel<uint64_t><<<blocks, 256, 0, st>>>(row_id_map, (const uint64_t *) rows, n, (uint64_t *) probs); break;
    default: return fail(PTB_ERR_ARG, "moe_rows_to_probs: element size %d", elem_bytes);
    }
    PTB_LAUNCH_CHECK("moe_rows_to_probs_kernel");
    return 0;
}

int ptb_zero_rows_after(const int64_t *counts, int64_t G, int64_t n_rows, int64_t row_bytes, void *out, ptb_stream_t stream) {
    PTB_REQUIRE(G >= 0 && n_rows >= 0 && row_bytes >= 0, PTB_ERR_ARG, "zero_rows_after: negative size");
    if (n_rows == 0 || row_bytes == 0) return 0;
    PTB_REQUIRE(out && (G == 0 || counts), PTB_ERR_ARG, "zero_rows_after: null pointer");
    zero_rows_after_kernel<<<148, 256, 0, (cudaStream_t) stream>>>(counts, G, n_rows, row_bytes, (uint8_t *) out);
    PTB_LAUNCH_CHECK("zero_rows_after_kernel");
    return 0;
}

int ptb_gather_rows_scaled(const void *in, int dtype, const int64_t *index, const float *weights, int64_t n_out,
                           int64_t n_in, int64_t H, void *out, ptb_stream_t stream) {
    PTB_REQUIRE(n_out >= 0 && n_in >= 0 && H >= 0, PTB_ERR_ARG, "gather_rows_scaled: negative size");
    if (n_out == 0 || H == 0) return 0;
    PTB_REQUIRE(index && weights && out && (n_in == 0 || in), PTB_ERR_ARG, "gather_rows_scaled: null pointer");
    const int blocks = (int) imin(cdiv<int64_t>(n_out, 8), 148 * 16);
    PTB_SWITCH_HP(dtype, T, (gather_rows_scaled_kernel<T><<<blocks, 256, 0, (cudaStream_t) stream>>>(
                                (const T *) in, index, weights, n_out, n_in, H, (T *) out)));
    PTB_LAUNCH_CHECK("gather_rows_scaled_kernel");
    return 0;
}

int ptb_unpermute_rows(const void *in, int dtype, const int32_t *row_id_map, const float *probs, int64_t T, int64_t E,
                       int64_t H, void *out, ptb_stream_t stream) {
    PTB_REQUIRE(T >= 0 && E >= 0 && H >= 0, PTB_ERR_ARG, "unpermute_rows: negative size");
    PTB_REQUIRE(E <= kMaxExperts, PTB_ERR_TOO_LARGE, "unpermute_rows: at most %d experts", kMaxExperts);
    if (T == 0 || H == 0) return 0;
    PTB_REQUIRE(out && row_id_map, PTB_ERR_ARG, "unpermute_rows: null pointer");
    const unsigned grid = (unsigned) cdiv<int64_t>(T, kUnpermWarps);
    PTB_SWITCH_HP(dtype, TT, if (unpermute_vec_ok<TT>(in, out, nullptr, H)) {
        unpermute_vec_kernel<TT, false><<<dim3(grid, unpermute_slices<TT>(H)), kUnpermWarps * 32, kUnpermWarps * 8 * (size_t) E,
                                          (cudaStream_t) stream>>>((const TT *) in, row_id_map, probs, T, E, H, (TT *) out, nullptr,
                                                                   nullptr);
        PTB_LAUNCH_CHECK("unpermute_vec_kernel");
        return 0;
    });
    PTB_SWITCH_HP(dtype, TT, (unpermute_kernel<TT, false><<<grid, kUnpermWarps * 32, 0, (cudaStream_t) stream>>>(
                                 (const TT *) in, row_id_map, probs, T, E, H, (TT *) out, nullptr, nullptr)));
    PTB_LAUNCH_CHECK("unpermute_kernel");
    return 0;
}

int ptb_unpermute_rows_bwd(const void *grad_out, int dtype, const void *fwd_in, const int32_t *row_id_map,
                           const float *probs, int64_t T, int64_t E, int64_t H, void *grad_in, float *grad_probs,
                           ptb_stream_t stream) {
    PTB_REQUIRE(T >= 0 && E >= 0 && H >= 0, PTB_ERR_ARG, "unpermute_rows_bwd: negative size");
    PTB_REQUIRE(E <= kMaxExperts, PTB_ERR_TOO_LARGE, "unpermute_rows_bwd: at most %d experts", kMaxExperts);
    if (T == 0 || H == 0) return 0;
    PTB_REQUIRE(grad_out && grad_in && row_id_map, PTB_ERR_ARG, "unpermute_rows_bwd: null pointer");
    PTB_REQUIRE(grad_probs == nullptr || fwd_in != nullptr, PTB_ERR_ARG, "unpermute_rows_bwd: grad_probs needs the forward rows");
    const unsigned grid = (unsigned) cdiv<int64_t>(T, kUnpermWarps);
    PTB_SWITCH_HP(dtype, TT, if (unpermute_vec_ok<TT>(grad_out, grad_in, grad_probs ? fwd_in : nullptr, H)) {
        const dim3 vgrid(grid, grad_probs != nullptr ? 1 : unpermute_slices<TT>(H));
        unpermute_vec_kernel<TT, true><<<vgrid, kUnpermWarps * 32, kUnpermWarps * 8 * (size_t) E, (cudaStream_t) stream>>>(
            (const TT *) grad_out, row_id_map, probs, T, E, H, (TT *) grad_in, (const TT *) fwd_in, grad_probs);
        PTB_LAUNCH_CHECK("unpermute_vec_kernel");
        return 0;
    });
    PTB_SWITCH_HP(dtype, TT, (unpermute_kernel<TT, true><<<grid, kUnpermWarps * 32, 0, (cudaStream_t) stream>>>(
                                 (const TT *) grad_out, row_id_map, probs, T, E, H, (TT *) grad_in, (const TT *) fwd_in,
                                 grad_probs)));
    PTB_LAUNCH_CHECK("unpermute_kernel");
    return 0;
}

#pragma GCC visibility pop
} // extern "C"
