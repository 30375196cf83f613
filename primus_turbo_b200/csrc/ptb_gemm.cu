// FP8 GEMM / grouped GEMM for sm_100a: TMA-fed shared-memory ring, tcgen05.mma with the
// accumulator in tensor memory, per-128-K-block scale promotion in registers, bf16/fp16 epilogue.
//
// Two forms of one kernel (CTAS): a 128 x 256 tile per CTA, or a 256 x 256 tile per pair of CTAs on neighbouring SMs
// (tcgen05 cta_group::2: each CTA loads its own 128 rows of A and half of B, and holds its own 128 output rows).
//
// One persistent CTA per SM, 384 threads:
//   warp 0      TMA producer (one lane): fills a ring of {A 128x128, B 256x128 or, in a pair, 128x128} FP8 tiles,
//               128-byte swizzled, either K-major or MN-major (transposed operands need no copy).
//   warp 1      MMA issuer (one lane; in a pair the first CTA's, for both): 4 x tcgen05.mma (N256 K32) per stage.  With blockwise
//               scales every 128-K block goes to one of two 256-column TMEM buffers with the
//               accumulate flag cleared, so each buffer holds one *partial* product.
//   warp 2      allocates / frees the 512 TMEM columns.
//   warps 4-11  two warpgroups (column halves 0-127 / 128-255): tcgen05.ld the partial, multiply by
//               a_scale*b_scale and accumulate in fp32 registers (or, for tensorwise / rowwise
//               scales, read the fully accumulated tile once), then convert and store.
// Tiles are assigned round-robin from a table derived on the device from the group offsets, so
// empty and skewed groups need no host synchronisation.  Every wait is bounded: on expiry the
// kernel records a status word, drains its own copies and leaves normally.
#include <cuda.h>

#include "ptb_common.cuh"

namespace ptb {
namespace {

constexpr int BM = 128, BK = 128;
constexpr int kABytes     = BM * BK;              // 16 KiB
constexpr int kMaxStages  = 8;
constexpr int kMaxAccBufs = 4;

// Compile-time geometry.  The tile is 128 x 256: eight promotion warps own 128 columns each, two
// 256-column TMEM buffers, 3 stages of 48 KiB.  (192- and 128-wide tiles were built and measured
// slower on every shape -- 8192^3 blockwise: 2044 TFLOP/s at 256, 1558 at 192 with twelve promotion
// warps, 1349 at 128 -- and are not compiled into the library.)
// DEEP = 1 trades the output staging buffer for more pipeline stages (plain stores in the epilogue).
//
// CTAS = 2.  What bounds the one-CTA tile once the scales are applied at the end is its shared memory: a 128-wide
// contraction block (8.4 MFLOP, 512 clocks of tensor pipe) writes and reads 48 KiB, 768 clocks at 128 bytes each; measured
// 855.  In a pair each CTA moves 32 KiB for the same work, because the tensor cores of both SMs read both halves of B:
// measured 730.
template <int BN, int DEEP, int CTAS> struct Geo {
    static_assert(BN == 256 && !(DEEP && CTAS == 2), "only these tiles are built");
    static constexpr int kSliceCols   = 128;                        // columns owned by one promotion warp
    static constexpr int kEpiWarps    = 4 * (BN / kSliceCols);      // 8
    static constexpr int kThreads     = 128 + 32 * kEpiWarps;
    static constexpr int kBBytes      = BN * BK / CTAS;
    static constexpr int kStageBytes  = kABytes + kBBytes;
    static constexpr int kStages      = CTAS == 2 ? 4 : 3 + DEEP;
    static constexpr int kAccBufs     = 512 / BN;
    static constexpr int kChunks      = kSliceCols / 32;            // 32-column TMEM loads per partial
    static constexpr int kWarpCBytes  = 32 * kSliceCols * 2;        // staging of one warp's 32-row slab (16-bit out)
    static constexpr int kCStageBytes = DEEP ? 0 : kEpiWarps * kWarpCBytes;
};
// Block scales reach the promotion warps through a shared-memory ring filled by a loader warp
// several contraction blocks ahead: one slot holds the 128 row scales of the tile's rows and up to
// 256 column scales (1-D x 1-D blocks) or one scale per column slice (1-D x 2-D blocks).
constexpr int kScaleSlots = 4;
constexpr int kSlotFloats = 128 + 256;
constexpr int kMaxGroups  = 1024;                 // tile table entries kept in shared memory
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s per wait, then give up

constexpr int kScaleTensor = 0, kScaleRow = 1, kScaleBlock2D = 2, kScaleBlock1D = 3, kScaleMX = 4;
// MX mode: E8M0 scale bytes, one per 32 contraction elements, travel global -> shared ring -> tensor
// memory (tcgen05.cp) and are applied by the block-scaled MMA itself; the accumulator then needs
// no promotion and one 256-column TMEM buffer leaves columns 256.. for the scale factors.
constexpr int kSfTmemCol0 = 256, kSfTmemColsPerSlot = 16; // per ring slot: 4 columns for A's 128 rows, 8 for B's 256
constexpr int kKindDense = 0, kKindGroupedRows = 1, kKindGroupedK = 2;

// status word written by a kernel whose wait ran out (0 = never happened)
__device__ int g_gemm_status = 0;

struct GemmArgs {
    CUtensorMap tm_a;
    CUtensorMap tm_b;
    CUtensorMap tm_c; // output, 16-bit elements, {64 columns, 32 rows} boxes (only when use_tma_store)
    int use_tma_store;
    int kind;
    int a_mn, b_mn; // 1: operand stored with the contraction axis strided (MN-major)
    uint32_t idesc;
    int M, N, K, G;
    int bn; // tile width the kernel was instantiated with
    int bm; // tile height: 128 per CTA of the tile
    int ctas; // CTAs that share a tile (1 or 2)
    int deep; // 1: variant without output staging
    int tiles_n;
    const int64_t *group_offs;
    void *c;
    int64_t ldc, c_group_stride;
    const float *a_scale;
    int64_t as_m, as_k;
    const float *b_scale;
    int64_t bs_g, bs_n, bs_k;
    // MX mode: scale bytes [rows][K / 32], row pitch in bytes (a multiple of 4)
    const uint8_t *a_sf, *b_sf;
    int64_t a_sf_ld, b_sf_ld;
};

// ---- PTX wrappers ------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// the same address in the shared memory of CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Arrival on a barrier of the pair's other CTA that publishes no write: it hands tensor memory whose reads have completed
// (tcgen05.wait::ld) back to the MMAs that overwrite it, and serves for nothing else.  A release at cluster scope waits for
// every outstanding access of the thread and tripled the time of the per-block modes.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void st_zero16_cluster(uint32_t cluster_addr) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(cluster_addr), "r"(0) : "memory");
}
__device__ __forceinline__ uint32_t cluster_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: false when the limit expired (the caller records the failure and leaves).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 256; ++i)
            if (mbar_try(bar, parity)) return true;
        if (globaltimer_ns() - t0 > kWaitLimitNs) return false;
    }
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *tm, uint32_t bar, int c0, int c1,
                                            int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
                 "%5}], [%2];" ::"r"(dst),
                 "l"(tm), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

// the same into this CTA's shared memory, with the barrier in either CTA of the pair (a shared::cluster address)
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *tm, uint32_t cluster_bar, int c0, int c1,
                                                 int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, "
                 "{%3, %4, %5}], [%2];" ::"r"(dst),
                 "l"(tm), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

__device__ __forceinline__ void tma_store_3d(const CUtensorMap *tm, uint32_t src, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(tm), "r"(src),
                 "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
// pulls a tensor map into the descriptor cache before the first copy that uses it
__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap *tm) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(tm) : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// 4-byte global -> shared copy that occupies no register while in flight
__device__ __forceinline__ void cp_async_f32(float *dst_smem, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst_smem)), "l"(src) : "memory");
}
// same, writing 0.0f instead when `valid` is false (the source is not read then)
__device__ __forceinline__ void cp_async_f32_zfill(float *dst_smem, const float *src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst_smem)), "l"(src),
                 "r"(valid ? 4u : 0u)
                 : "memory");
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// the barrier receives one arrival from this thread once all of its earlier cp.async copies have landed
__device__ __forceinline__ void cp_async_arrive_on(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

template <int CTAS = 1>
__device__ __forceinline__ void tc_mma_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    if constexpr (CTAS == 2) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                     "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                     : "memory");
    } else {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                     "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                     : "memory");
    }
}
// block-scaled FP8 MMA: one E8M0 scale per 32 contraction elements of every A row and B row, read from
// tensor memory; the byte of the 32-bit scale cell to use is part of the instruction descriptor
__device__ __forceinline__ void tc_mma_mxf8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%4], [%5], p;\n\t}" ::"r"(d_tmem),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(sfa_tmem), "r"(sfb_tmem), "r"(accumulate)
                 : "memory");
}
// 32 rows x 16 bytes of shared memory -> 4 TMEM columns of lanes 0-31, repeated in all four lane quarters
__device__ __forceinline__ void tc_cp_sf(uint32_t dst_tmem, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(dst_tmem), "l"(sdesc) : "memory");
}
// Arrives on `bar` once the MMAs issued so far have retired; a pair's issuer arrives on that barrier of both CTAs.
template <int CTAS = 1> __device__ __forceinline__ void tc_commit(uint32_t bar) {
    if constexpr (CTAS == 2) {
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                     "h"((uint16_t) 3)
                     : "memory");
        return;
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                   "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                   "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, 128-byte swizzle, version 1 (sm_100).
//   K-major tile  [rows][128 B]: 8-row groups 1024 B apart (SBO); LBO unused.
//   MN-major tile [k rows][128 B of M/N]: 8-k groups 1024 B apart (SBO), next 128-wide M/N chunk LBO apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t) ((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t) ((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t) ((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t) 1 << 46; // descriptor version
    d |= (uint64_t) 2 << 61; // SWIZZLE_128B
    return d;
}

// Shared-memory descriptor of a 128-row scale-factor atom for tcgen05.cp: no swizzle, rows of 16 bytes,
// 8-row groups 128 bytes apart.
__device__ __forceinline__ uint64_t make_sf_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t) ((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t) (128u >> 4) << 32;
    d |= (uint64_t) 1 << 46;
    return d;
}

// ---- tile schedule -----------------------------------------------------------------------------
struct Tile {
    int m0;        // first output row (absolute row of C / of the grouped A)
    int m_end;     // first row that must not be stored
    int n0;        // first output column
    int g;         // group (0 for dense)
    int k_row0;    // first contraction row (variable-K) else 0
    int num_kb;    // 128-wide contraction blocks
    int k_tail;    // variable-K only: valid rows of the last block when the group length is not a multiple of 128, else 0
};

struct __align__(16) SharedCtl {
    float scale_ring[kScaleSlots * kSlotFloats]; // per contraction block: 128 row scales, then the column scales
    uint64_t sc_full[kScaleSlots];
    uint64_t sc_empty[kScaleSlots];
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t cut[kMaxStages]; // pairs, in the first CTA: both CTAs' copies of a block that reaches past its group have landed
    uint64_t tmem_full[kMaxAccBufs];
    uint64_t tmem_empty[kMaxAccBufs];
    uint32_t tmem_base;
    uint32_t sf_batches_done; // MX scale loaders: batches of four blocks whose slots have been claimed and filled
    int total_tiles;
    int sched_q, sched_rem; // grid stride = sched_q * tiles_n + sched_rem
    int tile_prefix[kMaxGroups + 1];
    int group_offs[kMaxGroups + 1]; // copy of the device offsets: the schedule never waits on global memory
};

// Walks the tiles u, u + units, ... of one CTA or pair (u of units).  The linear index is split
// into its coordinates once, with divisions, in the constructor; every later tile is reached by
// adding the (pre-split) grid stride and carrying, because each role warp pays for the walk on its
// critical path once per tile and short-K tiles (wgrad) last only a few thousand cycles.
struct Schedule {
    const GemmArgs &a;
    const SharedCtl *ctl; // loop invariants are re-read from shared / constant memory instead of held in registers
    int lin;
    int p0, p1, p2; // dense: (band, index in band, -); grouped rows: (m-tile, n-tile, group cursor);
                    // grouped variable-K: (group, m-tile, n-tile)

    __device__ Schedule(const GemmArgs &args, const SharedCtl *c) : a(args), ctl(c), lin(blockIdx.x / args.ctas) {
        p0 = p1 = p2 = 0;
        if (lin >= ctl->total_tiles) return;
        if (a.kind == kKindDense) {
            const int band = 8 * a.tiles_n;
            p0 = lin / band;
            p1 = lin - p0 * band;
        } else if (a.kind == kKindGroupedRows) {
            p0 = lin / a.tiles_n;
            p1 = lin - p0 * a.tiles_n;
        } else {
            const int per_g = ((a.M + a.bm - 1) / a.bm) * a.tiles_n;
            p0          = lin / per_g;
            const int r = lin - p0 * per_g;
            p1 = r / a.tiles_n;
            p2 = r - p1 * a.tiles_n;
        }
    }

    // Emits the current tile and steps to the CTA's next one; false when the CTA has no tile left.
    __device__ bool get(Tile &o) {
        if (lin >= ctl->total_tiles) return false;
        const int step = gridDim.x / a.ctas, tiles_m = (a.M + a.bm - 1) / a.bm;
        const int *offs = ctl->group_offs;
        if (a.kind == kKindDense) {
            // bands of 8 row-tiles, rows fastest inside a band: neighbouring CTAs share B columns
            // and a narrow band of A rows.
            int rows;
            for (;;) {
                rows = min(8, tiles_m - 8 * p0);
                const int sz = rows * a.tiles_n;
                if (p1 < sz) break;
                p1 -= sz;
                ++p0;
            }
            const int nt = rows == 8 ? (p1 >> 3) : p1 / rows;
            const int mt = 8 * p0 + (p1 - nt * rows);
            o.m0 = mt * a.bm; o.m_end = a.M; o.n0 = nt * a.bn; o.g = 0; o.k_row0 = 0;
            o.num_kb = (a.K + BK - 1) / BK; o.k_tail = 0;
            p1 += step;
        } else if (a.kind == kKindGroupedRows) {
            const int *tile_prefix = ctl->tile_prefix;
            while (tile_prefix[p2 + 1] <= p0) ++p2;
            const int g  = p2;
            const int lo = offs[g], hi = offs[g + 1];
            o.m0 = lo + (p0 - tile_prefix[g]) * a.bm; o.m_end = hi; o.n0 = p1 * a.bn; o.g = g;
            o.k_row0 = 0; o.num_kb = (a.K + BK - 1) / BK; o.k_tail = 0;
            p1 += ctl->sched_rem;
            p0 += ctl->sched_q;
            if (p1 >= a.tiles_n) { p1 -= a.tiles_n; ++p0; }
        } else {
            const int lo = offs[p0], hi = offs[p0 + 1];
            o.m0 = p1 * a.bm; o.m_end = a.M; o.n0 = p2 * a.bn; o.g = p0; o.k_row0 = lo;
            o.num_kb = (hi - lo + BK - 1) / BK;
            o.k_tail = (hi - lo) % BK;
            p2 += ctl->sched_rem;
            p1 += ctl->sched_q;
            if (p2 >= a.tiles_n) { p2 -= a.tiles_n; ++p1; }
            while (p1 >= tiles_m) { p1 -= tiles_m; ++p0; }
        }
        lin += step;
        return true;
    }
};

template <typename OutT> struct Pack8;
template <> struct Pack8<__nv_bfloat16> {
    static __device__ __forceinline__ uint4 pack(const float *v) {
        uint4 o;
        __nv_bfloat162 t;
        t = __floats2bfloat162_rn(v[0], v[1]); o.x = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2bfloat162_rn(v[2], v[3]); o.y = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2bfloat162_rn(v[4], v[5]); o.z = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2bfloat162_rn(v[6], v[7]); o.w = *reinterpret_cast<uint32_t *>(&t);
        return o;
    }
    static __device__ __forceinline__ void store(__nv_bfloat16 *p, const float *v) {
        uint4 o;
        __nv_bfloat162 t;
        t = __floats2bfloat162_rn(v[0], v[1]); o.x = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2bfloat162_rn(v[2], v[3]); o.y = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2bfloat162_rn(v[4], v[5]); o.z = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2bfloat162_rn(v[6], v[7]); o.w = *reinterpret_cast<uint32_t *>(&t);
        *reinterpret_cast<uint4 *>(p) = o;
    }
};
template <> struct Pack8<__half> {
    static __device__ __forceinline__ uint4 pack(const float *v) {
        uint4 o;
        __half2 t;
        t = __floats2half2_rn(v[0], v[1]); o.x = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2half2_rn(v[2], v[3]); o.y = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2half2_rn(v[4], v[5]); o.z = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2half2_rn(v[6], v[7]); o.w = *reinterpret_cast<uint32_t *>(&t);
        return o;
    }
    static __device__ __forceinline__ void store(__half *p, const float *v) {
        uint4 o;
        __half2 t;
        t = __floats2half2_rn(v[0], v[1]); o.x = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2half2_rn(v[2], v[3]); o.y = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2half2_rn(v[4], v[5]); o.z = *reinterpret_cast<uint32_t *>(&t);
        t = __floats2half2_rn(v[6], v[7]); o.w = *reinterpret_cast<uint32_t *>(&t);
        *reinterpret_cast<uint4 *>(p) = o;
    }
};
template <> struct Pack8<float> {
    static __device__ __forceinline__ uint4 pack(const float *) { return make_uint4(0, 0, 0, 0); } // 16-bit outputs only
    static __device__ __forceinline__ void store(float *p, const float *v) {
        *reinterpret_cast<float4 *>(p)     = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4 *>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
};


// The last block of an unpadded variable-K group reaches into the next group's rows (or past the last group): clear
// those contraction rows in both MN-major operand tiles, so that whatever bytes lie there -- FP8 NaN patterns
// included -- add nothing.  Rows up to `end` only: with tensorwise and rowwise scales the MMA steps (of 32 rows) that hold
// no valid row are not issued.  A contraction row is 128 bytes in the A tile and in each 128-column part of the B tile;
// the swizzle only permutes bytes inside a row.  One warp.
template <int B_PARTS> __device__ __forceinline__ void clear_tail_rows(uint8_t *a_tile, int k_tail, int end, int lane) {
    for (int off = k_tail * 128 + lane * 16; off < end * 128; off += 32 * 16) {
#pragma unroll
        for (int p = 0; p <= B_PARTS; ++p) *reinterpret_cast<uint4 *>(a_tile + p * 16384 + off) = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// The same for a pair's block: the tiles of this CTA and, through `peer` (the same address in the other CTA), of the other.
template <int B_PARTS> __device__ __forceinline__ void clear_tail_rows_pair(uint8_t *a_tile, uint32_t peer, int k_tail, int end, int lane) {
    for (int off = k_tail * 128 + lane * 16; off < end * 128; off += 32 * 16) {
#pragma unroll
        for (int p = 0; p <= B_PARTS; ++p) {
            st_zero16_cluster(peer + p * 16384 + off);
            *reinterpret_cast<uint4 *>(a_tile + p * 16384 + off) = make_uint4(0, 0, 0, 0);
        }
    }
    asm volatile("fence.proxy.async;" ::: "memory");
}

template <int SCALE, typename OutT, int BN, int DEEP, int CTAS>
__global__ void __launch_bounds__(Geo<BN, DEEP, CTAS>::kThreads, 1) fp8_gemm_kernel(const __grid_constant__ GemmArgs args) {
    using G_ = Geo<BN, DEEP, CTAS>;
    static_assert(CTAS == 1 || SCALE == kScaleTensor || SCALE == kScaleRow, "block scales run one CTA per tile");
    constexpr int kStages = G_::kStages, kStageBytes = G_::kStageBytes, kThreads = G_::kThreads;
    constexpr int kAccBufs = (SCALE == kScaleMX) ? 1 : G_::kAccBufs, kWgCols = G_::kSliceCols, kChunks = G_::kChunks;
    constexpr int kCStageBytes = G_::kCStageBytes, kEpiWarps = G_::kEpiWarps;
    extern __shared__ uint8_t smem_raw[];
    // tiles need 1024-byte alignment for the 128-byte swizzle
    uint8_t *smem  = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *c_stage = smem + kStages * kStageBytes;
    SharedCtl *ctl   = reinterpret_cast<SharedCtl *>(c_stage + kCStageBytes);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = smem_u32(smem);
    const int rank     = CTAS == 2 ? (int) cluster_cta_rank() : 0; // this CTA's half of the tile
    const bool leader  = rank == 0;
    constexpr bool kPerBlock = (SCALE == kScaleBlock2D || SCALE == kScaleBlock1D);
    constexpr bool kSkipSteps = SCALE == kScaleTensor || SCALE == kScaleRow; // the modes with unpadded variable-K groups

    // ---- set-up: barriers, tile table, tensor memory -------------------------------------------
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&ctl->full[s]), 1);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
            mbar_init(smem_u32(&ctl->cut[s]), 1);
        }
        for (int b = 0; b < kAccBufs; ++b) {
            mbar_init(smem_u32(&ctl->tmem_full[b]), 1);
            mbar_init(smem_u32(&ctl->tmem_empty[b]), CTAS * kEpiWarps); // one arrival per promotion warp
        }
        for (int b = 0; b < kScaleSlots; ++b) {
            mbar_init(smem_u32(&ctl->sc_full[b]), 32);         // every loader lane, after its own copies
            // one arrival per promotion warp; in MX mode the MMA issuer's commit frees the slot
            mbar_init(smem_u32(&ctl->sc_empty[b]), SCALE == kScaleMX ? 1 : kEpiWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (threadIdx.x == 64) {
        tma_prefetch_map(&args.tm_a);
        tma_prefetch_map(&args.tm_b);
        if (args.use_tma_store) tma_prefetch_map(&args.tm_c);
    }
    if (threadIdx.x == 32) {
        ctl->sf_batches_done = 0;
        ctl->sched_q   = (int) (gridDim.x / CTAS) / args.tiles_n;
        ctl->sched_rem = (int) (gridDim.x / CTAS) % args.tiles_n;
    }
    // The pair's tensor memory is allocated by both CTAs together, and barriers of one are signalled by the other: both CTAs
    // run and have set up their barriers before either goes on.
    if constexpr (CTAS == 2) cluster_sync();
    if (warp == 2) {
        if constexpr (CTAS == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                             smem_u32(&ctl->tmem_base))
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                             smem_u32(&ctl->tmem_base))
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    grid_dep_begin(); // everything above touches no global memory
    if (args.kind != kKindDense) {
        for (int g = threadIdx.x; g <= args.G; g += kThreads) ctl->group_offs[g] = (int) args.group_offs[g];
    }
    if (args.kind == kKindGroupedRows) {
        // cumulative row tiles per group; one warp scans (G <= kMaxGroups, checked on the host)
        if (warp == 3) {
            int run = 0;
            for (int base = 0; base < args.G; base += 32) {
                const int g = base + lane;
                int cnt     = 0;
                if (g < args.G) cnt = (int) ((args.group_offs[g + 1] - args.group_offs[g] + CTAS * BM - 1) / (CTAS * BM));
                int inc = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    int n = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += n;
                }
                if (g < args.G) ctl->tile_prefix[g + 1] = run + inc;
                run += __shfl_sync(0xffffffffu, inc, 31);
            }
            if (lane == 0) {
                ctl->tile_prefix[0] = 0;
                ctl->total_tiles    = run * args.tiles_n;
            }
        }
    } else if (threadIdx.x == 0) {
        const int tiles_m = (args.M + CTAS * BM - 1) / (CTAS * BM);
        ctl->total_tiles  = (args.kind == kKindDense ? 1 : args.G) * tiles_m * args.tiles_n;
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (CTAS == 2) cluster_sync(); // the other CTA has its tensor memory too
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;

    if (warp < 4) {
        // register split between the helper warpgroup and the two promotion warpgroups: the 1-D x 1-D
        // promotion needs every register it can get, the other modes leave more to the MMA issuer
        // (in MX mode the scale loader keeps four blocks of scale words in registers and the epilogue holds no
        // promotion state, so the split moves the other way).  Neither side may spill in a loop: with the shared memory all
        // taken the L1 is tiny and a spilled register comes back from L2.
        if constexpr (SCALE == kScaleBlock1D) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        else if constexpr (SCALE == kScaleBlock2D) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        else if constexpr (SCALE == kScaleMX) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp == 0 && lane == 0) {
            // ================= TMA producer =================
            Schedule sched(args, ctl);
            Tile t;
            uint32_t it = 0; // ring position over the whole kernel
            uint32_t cut = 0, cut_ph = 0; // pairs, a bit per stage: the last copies signal `cut`; the phase of that barrier
            bool ok     = true;
            while (ok && sched.get(t)) {
                const int gb = (args.kind == kKindGroupedRows) ? t.g : 0;
                for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
                    const int s = it % kStages;
                    const uint32_t ph = (it / kStages) & 1;
                    if (!mbar_wait(smem_u32(&ctl->empty[s]), ph ^ 1)) { ok = false; break; }
                    const uint32_t full = smem_u32(&ctl->full[s]);
                    const uint32_t sa = smem_base + s * kStageBytes, sb = sa + kABytes;
                    const int k = t.k_row0 + kb * BK;
                    if constexpr (CTAS == 2) {
                        // Both CTAs' copies complete on the first CTA's barrier; on `cut` for a block with rows to clear, whose
                        // `full` warp 3 completes.  A half of A that holds no row of the tile is not fetched: its
                        // products are never read.
                        const int m0 = t.m0 + rank * BM, n0 = t.n0 + rank * (BN / 2);
                        const bool has_a = m0 < t.m_end, past = t.k_tail != 0 && kb == t.num_kb - 1;
                        const uint32_t mine = past ? smem_u32(&ctl->cut[s]) : full, bar = map_to_cta(mine, 0);
                        if (leader) mbar_expect_tx(mine, m0 + BM < t.m_end ? 2 * kStageBytes : 2 * kStageBytes - kABytes);
                        cut    = past ? cut | 1u << s : cut & ~(1u << s);
                        cut_ph ^= past ? 1u << s : 0u;
                        if (has_a) {
                            if (args.a_mn) tma_load_3d_pair(sa, &args.tm_a, bar, m0, k, 0);
                            else           tma_load_3d_pair(sa, &args.tm_a, bar, k, m0, 0);
                        }
                        if (args.b_mn) tma_load_3d_pair(sb, &args.tm_b, bar, n0, k, gb);
                        else           tma_load_3d_pair(sb, &args.tm_b, bar, k, n0, gb);
                        continue;
                    }
                    mbar_expect_tx(full, kStageBytes);
                    if (args.a_mn) tma_load_3d(sa, &args.tm_a, full, t.m0, k, 0);
                    else           tma_load_3d(sa, &args.tm_a, full, k, t.m0, 0);
                    if (args.b_mn) {
                        tma_load_3d(sb, &args.tm_b, full, t.n0, k, gb);
                        tma_load_3d(sb + 16384, &args.tm_b, full, t.n0 + 128, k, gb); // MN-major boxes are 128 columns wide
                    } else {
                        tma_load_3d(sb, &args.tm_b, full, k, t.n0, gb);
                    }
                }
            }
            if (!ok) {
                atomicExch(&g_gemm_status, 1);
                // let the copies already issued land before the CTA releases its shared memory (a pair's second CTA
                // finds its copies' barrier in the first; the pair leaves together, after the first has waited)
                if (CTAS == 2 && !leader) it = 0;
                const uint32_t back = it < (uint32_t) kStages ? it : (uint32_t) kStages;
                for (uint32_t j = 1; j <= back; ++j) {
                    const uint32_t q = it - j, s = q % kStages;
                    if (CTAS == 2 && (cut >> s & 1)) mbar_wait(smem_u32(&ctl->cut[s]), (cut_ph >> s & 1) ^ 1);
                    else mbar_wait(smem_u32(&ctl->full[s]), (q / kStages) & 1);
                }
            }
        } else if (warp == 1 && leader) {
            // ================= MMA issuer (whole warp walks the schedule, lane 0 issues) =================
            Schedule sched(args, ctl);
            Tile t;
            uint32_t it = 0, acc_it = 0;
            bool ok     = true;
            const uint32_t a_lbo = 0, a_sbo = 1024, a_step = args.a_mn ? 4096u : 32u;
            const uint32_t b_lbo = args.b_mn && CTAS == 1 ? 16384u : 0u, b_sbo = 1024;
            const uint32_t b_step = args.b_mn ? 4096u : 32u;
            while (ok && sched.get(t)) {
                for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
                    const int s = it % kStages;
                    const uint32_t ph = (it / kStages) & 1;
                    const bool new_acc = kPerBlock || kb == 0;
                    const uint32_t buf = acc_it % kAccBufs;
                    if (new_acc) {
                        if (!mbar_wait(smem_u32(&ctl->tmem_empty[buf]), ((acc_it / kAccBufs) & 1) ^ 1)) { ok = false; break; }
                    }
                    if (!mbar_wait(smem_u32(&ctl->full[s]), ph)) { ok = false; break; }
                    const int slot = it % kScaleSlots;
                    if constexpr (SCALE == kScaleMX) {
                        if (!mbar_wait(smem_u32(&ctl->sc_full[slot]), (it / kScaleSlots) & 1)) { ok = false; break; }
                    }
                    uint8_t *a_tile = smem + s * kStageBytes;
                    const bool past = t.k_tail != 0 && kb == t.num_kb - 1; // the block reaches past its group
                    if (CTAS == 1 && past) // (a pair's warp 3 has done it)
                        clear_tail_rows<G_::kBBytes / 16384>(a_tile, t.k_tail, kSkipSteps ? (t.k_tail + 31) & ~31 : BK, lane);
                    __syncwarp();
                    tc_fence_after();
                    if (lane == 0) {
                        const uint32_t sa = smem_base + s * kStageBytes, sb = sa + kABytes;
                        const uint32_t d  = tmem_base + buf * BN;
                        const uint64_t ad = make_smem_desc(sa, a_lbo, a_sbo);
                        const uint64_t bd = make_smem_desc(sb, b_lbo, b_sbo);
                        if constexpr (SCALE == kScaleMX) {
                            // this block's scale bytes: three 512-byte atoms (A rows, B rows 0-127, B rows 128-255)
                            const uint32_t sf_smem = smem_u32(&ctl->scale_ring[slot * kSlotFloats]);
                            const uint32_t sf_tmem = tmem_base + kSfTmemCol0 + slot * kSfTmemColsPerSlot;
                            tc_cp_sf(sf_tmem, make_sf_desc(sf_smem));
                            tc_cp_sf(sf_tmem + 4, make_sf_desc(sf_smem + 512));
                            tc_cp_sf(sf_tmem + 8, make_sf_desc(sf_smem + 1024));
#pragma unroll
                            for (int j = 0; j < BK / 32; ++j) {
                                const uint32_t accumulate = (j > 0 || !new_acc) ? 1u : 0u;
                                // byte j of each scale cell belongs to the j-th 32-wide slice of the block
                                const uint32_t idesc = args.idesc | ((uint32_t) j << 29) | ((uint32_t) j << 4);
                                tc_mma_mxf8(d, ad + (uint64_t) ((a_step * j) >> 4), bd + (uint64_t) ((b_step * j) >> 4), idesc,
                                            sf_tmem, sf_tmem + 4, accumulate);
                            }
                            tc_commit(smem_u32(&ctl->sc_empty[slot])); // scale slot reusable once copies and MMAs retire
                        } else if (kSkipSteps && past) {
#pragma unroll 1
                            for (int j = 0; 32 * j < t.k_tail; ++j)
                                tc_mma_f8<CTAS>(d, ad + (uint64_t) ((a_step * j) >> 4), bd + (uint64_t) ((b_step * j) >> 4), args.idesc,
                                                (j > 0 || !new_acc) ? 1u : 0u);
                        } else {
#pragma unroll
                            for (int j = 0; j < BK / 32; ++j) {
                                const uint32_t accumulate = (j > 0 || !new_acc) ? 1u : 0u;
                                tc_mma_f8<CTAS>(d, ad + (uint64_t) ((a_step * j) >> 4), bd + (uint64_t) ((b_step * j) >> 4),
                                                args.idesc, accumulate);
                            }
                        }
                        tc_commit<CTAS>(smem_u32(&ctl->empty[s])); // stage reusable once these MMAs retire
                    }
                    const bool last = kPerBlock || kb == t.num_kb - 1;
                    if (last) {
                        if (lane == 0) tc_commit<CTAS>(smem_u32(&ctl->tmem_full[buf]));
                        ++acc_it;
                    }
                }
            }
            if (!ok && lane == 0) atomicExch(&g_gemm_status, 2);
        } else if (CTAS == 2 && warp == 3) {
            // ================= pairs, first CTA: blocks that reach past their group =================
            // The MMA reads both CTAs' tiles, and this warp clears both, so that the writes, the proxy fence, the stage's
            // barrier and the MMA all lie in one CTA.  (The second CTA clearing its own half has to hand it over with a
            // release and an acquire at cluster scope: wgrad of 64 groups of 60 rows on average, 2048 x 2048: 152 us.)
            Schedule sched(args, ctl);
            Tile t;
            uint32_t it = 0, ph = 0; // ph: a bit per stage
            while (leader && sched.get(t)) {
                it += t.num_kb;
                if (t.k_tail == 0) continue;
                const int s = (it - 1) % kStages; // the tile's last block
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->cut[s]), ph >> s & 1))) { // the warp leaves as one
                    if (lane == 0) atomicExch(&g_gemm_status, 2);
                    break;
                }
                ph ^= 1u << s;
                clear_tail_rows_pair<G_::kBBytes / 16384>(smem + s * kStageBytes, map_to_cta(smem_base + s * kStageBytes, 1), t.k_tail,
                                                            (t.k_tail + 31) & ~31, lane);
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctl->full[s]));
            }
        } else if (warp == 3 || (SCALE == kScaleMX && warp == 2)) {
            // ================= scale loader (1-D x 1-D block scales; MX: warps 2 and 3) =================
            // Copies each contraction block's row and column scales into the ring with cp.async; the
            // slot's barrier hears from every lane when that lane's copies have landed, so neither this
            // warp nor the promotion warps ever hold a register waiting on a scale load from global
            // memory.  (With 1-D x 2-D blocks a thread needs two scalars per block and fetches them
            // itself two blocks ahead: measured faster than a ring there.)
            if constexpr (SCALE == kScaleBlock1D) {
                Schedule sched(args, ctl);
                Tile t;
                uint32_t it = 0;
                bool ok     = true;
                while (ok && sched.get(t)) {
                    const int kb_base = t.k_row0 / BK;
                    for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
                        const int slot = it % kScaleSlots;
                        if (!mbar_wait(smem_u32(&ctl->sc_empty[slot]), ((it / kScaleSlots) & 1) ^ 1)) { ok = false; break; }
                        float *dst         = &ctl->scale_ring[slot * kSlotFloats];
                        const float *a_src = args.a_scale + (int64_t) (kb_base + kb) * args.as_k;
#pragma unroll
                        for (int i = 0; i < BM / 32; ++i) {
                            const int r = min(t.m0 + i * 32 + lane, t.m_end - 1); // rows past the group are never stored
                            cp_async_f32(dst + i * 32 + lane, a_src + (int64_t) r * args.as_m);
                        }
                        const float *b_src = args.b_scale + (int64_t) (kb_base + kb) * args.bs_k;
#pragma unroll
                        for (int i = 0; i < BN / 32; ++i) {
                            const int c = t.n0 + i * 32 + lane;
                            cp_async_f32_zfill(dst + 128 + i * 32 + lane, b_src + (int64_t) min(c, args.N - 1) * args.bs_n,
                                               c < args.N);
                        }
                        cp_async_arrive_on(smem_u32(&ctl->sc_full[slot]));
                    }
                }
                cp_async_wait_all(); // nothing of this warp's is in flight when the CTA tears down
                if (!ok && lane == 0) atomicExch(&g_gemm_status, 4);
            }
            if constexpr (SCALE == kScaleMX) {
                // Gathers the scale bytes of four contraction blocks at a time -- one aligned 16-byte load per
                // operand row (a block's four 32-wide slices are one 32-bit word) -- and lays each block out
                // as tcgen05.cp wants it: row r of a 128-row atom at byte 16 * (r % 32) + 4 * (r / 32), so a
                // lane's four rows (lane, lane + 32, ...) are one 16-byte store.  Warps 2 and 3 take the batches
                // of four blocks in turn: while one waits for ring slots to store its batch, the other's loads
                // for the next batch are already in flight, so the global round trip is never exposed (one
                // loader warp left the tensor pipe idle for it once per four blocks: 37 % active).
                Schedule sched(args, ctl);
                Tile t;
                uint32_t it = 0, batch = 0;
                bool ok     = true;
                const uint32_t mine = warp & 1; // warp 2: even batches, warp 3: odd batches
                // rows of 16 scale bytes can be read with one vector load when the pitch and base allow it
                const bool vec = (args.a_sf_ld % 16 == 0) && (args.b_sf_ld % 16 == 0) &&
                                 ((reinterpret_cast<uintptr_t>(args.a_sf) | reinterpret_cast<uintptr_t>(args.b_sf)) & 15u) == 0;
                while (ok && sched.get(t)) {
                    int row[12]; // operand rows whose scale words this lane moves (clamped: rows past the end are never stored)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        row[i]     = min(t.m0 + lane + 32 * i, t.m_end - 1);
                        row[4 + i] = min(t.n0 + lane + 32 * i, args.N - 1);
                        row[8 + i] = min(t.n0 + 128 + lane + 32 * i, args.N - 1);
                    }
                    // per-expert weights: B's scale rows follow the groups; variable-K groups: the scale bytes of
                    // contraction rows [k_row0, ...) start k_row0 / 32 bytes into every operand row
                    const int64_t b_row0 = (args.kind == kKindGroupedRows) ? (int64_t) t.g * args.N : 0;
                    const int k_byte0    = t.k_row0 / 32;
                    const bool vec_t     = vec && ((k_byte0 & 15) == 0);
                    uint4 w[12];
                    int loaded_kb = -1; // first block of the batch whose words are in w
                    auto load_batch = [&](int kb0) {
#pragma unroll
                        for (int i = 0; i < 12; ++i) {
                            const uint8_t *src = (i < 4 ? args.a_sf + (int64_t) row[i] * args.a_sf_ld
                                                        : args.b_sf + (b_row0 + row[i]) * args.b_sf_ld) + k_byte0 + 4 * kb0;
                            if (vec_t && kb0 + 4 <= t.num_kb) {
                                w[i] = *reinterpret_cast<const uint4 *>(src);
                            } else {
                                const uint32_t *s32 = reinterpret_cast<const uint32_t *>(src);
                                w[i].x = s32[0];
                                w[i].y = kb0 + 1 < t.num_kb ? s32[1] : 0u;
                                w[i].z = kb0 + 2 < t.num_kb ? s32[2] : 0u;
                                w[i].w = kb0 + 3 < t.num_kb ? s32[3] : 0u;
                            }
                        }
                        loaded_kb = kb0;
                    };
                    for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
                        const bool start = (kb & 3) == 0;
                        if (start) ++batch;
                        const bool own = ((batch - 1) & 1) == mine;
                        if (start) {
                            // own batch: fetch it unless it is already here; the other warp's batch: fetch the one
                            // after it (batches alternate, so that one is this warp's) before waiting on the ring
                            if (own) {
                                if (loaded_kb != kb) load_batch(kb);
                            } else if (kb + 4 < t.num_kb) {
                                load_batch(kb + 4);
                            }
                        }
                        if (!own) continue;
                        // Hand-over between the two warps: a batch's slots are claimed only after the previous
                        // batch's owner has passed all of its waits.  A parity wait tells "this phase is over"
                        // from "the previous phase is over" only for a waiter within one phase of the barrier;
                        // the owner of batch b last waited on these slots for batch b - 2, and without the
                        // hand-over it could find a slot's barrier still one phase back, pass at once and
                        // overwrite a block the tensor cores have not read.
                        if (start) {
                            const volatile uint32_t *done = &ctl->sf_batches_done;
                            if (*done != batch - 1) {
                                const uint64_t t0 = globaltimer_ns();
                                while (*done != batch - 1) {
                                    __nanosleep(40);
                                    if (globaltimer_ns() - t0 > kWaitLimitNs) { ok = false; break; }
                                }
                                if (!ok) break;
                            }
                        }
                        const int slot = it % kScaleSlots;
                        if (!mbar_wait(smem_u32(&ctl->sc_empty[slot]), ((it / kScaleSlots) & 1) ^ 1)) { ok = false; break; }
                        const uint32_t dst = smem_u32(&ctl->scale_ring[slot * kSlotFloats]) + lane * 16;
                        const int q = kb & 3;
#define PTB_SFW(i) (q == 0 ? w[i].x : q == 1 ? w[i].y : q == 2 ? w[i].z : w[i].w)
                        st_shared_v4(dst, make_uint4(PTB_SFW(0), PTB_SFW(1), PTB_SFW(2), PTB_SFW(3)));
                        st_shared_v4(dst + 512, make_uint4(PTB_SFW(4), PTB_SFW(5), PTB_SFW(6), PTB_SFW(7)));
                        st_shared_v4(dst + 1024, make_uint4(PTB_SFW(8), PTB_SFW(9), PTB_SFW(10), PTB_SFW(11)));
#undef PTB_SFW
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // tcgen05.cp reads through the async proxy
                        mbar_arrive(smem_u32(&ctl->sc_full[slot]));
                        if ((kb & 3) == 3 || kb == t.num_kb - 1) {
                            // last block of this warp's batch: the other warp may claim the slots that follow
                            __syncwarp();
                            if (lane == 0) *reinterpret_cast<volatile uint32_t *>(&ctl->sf_batches_done) = batch;
                        }
                    }
                }
                if (!ok) {
                    // release a partner that may be waiting for the hand-over; it will run into its own limits
                    if (lane == 0) {
                        *reinterpret_cast<volatile uint32_t *>(&ctl->sf_batches_done) = 0xffffffffu;
                        atomicExch(&g_gemm_status, 4);
                    }
                }
            }
        }
    } else {
        if constexpr (SCALE == kScaleBlock1D) asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        else if constexpr (SCALE == kScaleBlock2D) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        else if constexpr (SCALE == kScaleMX) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        else asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        // ================= promotion + epilogue warpgroups =================
        const int wg   = (warp - 4) >> 2;         // column slice of the tile this warp owns
        const int quad = warp & 3;                // TMEM lane quadrant this warp may read
        const int row_in_tile = quad * 32 + lane;
            OutT *cbase           = reinterpret_cast<OutT *>(args.c);

        if (args.kind == kKindGroupedRows) {
            // zero the rows past the last group (output is allocated for M rows)
            const int64_t first = args.group_offs[args.G];
            const int64_t nvec  = (int64_t) (args.M - first) * args.N;
            const int64_t e0    = (int64_t) blockIdx.x * (32 * kEpiWarps) + (threadIdx.x - 128);
            for (int64_t e = e0; e < nvec; e += (int64_t) gridDim.x * (32 * kEpiWarps)) {
                const int64_t r = first + e / args.N, c = e % args.N;
                cbase[r * args.ldc + c] = from_f32<OutT>(0.0f);
            }
        }

        Schedule sched(args, ctl);
        Tile t;
        uint32_t acc_it = 0;
        bool ok         = true;
        const bool vec_store = ((args.ldc * sizeof(OutT)) % 16 == 0) && ((reinterpret_cast<uintptr_t>(args.c) & 15u) == 0) &&
                               ((args.c_group_stride * sizeof(OutT)) % 16 == 0);
        const bool tma_store  = (sizeof(OutT) == 2) && args.use_tma_store && !DEEP;
        uint8_t *my_stage     = c_stage + (warp - 4) * G_::kWarpCBytes;
        const uint32_t stage_u32 = smem_u32(my_stage);
        bool store_pending    = false;
        float acc[kWgCols];
        while (ok && sched.get(t)) {
            const int gb      = (args.kind == kKindGroupedRows) ? t.g : 0;
            if constexpr (CTAS == 2) t.m0 += rank * BM; // this CTA's rows (none, where the group ends before them)
            const int row     = t.m0 + row_in_tile;
            const int col0    = t.n0 + wg * kWgCols;
            const int segs    = kPerBlock ? t.num_kb : (t.num_kb > 0 ? 1 : 0);
#pragma unroll
            for (int j = 0; j < kWgCols; ++j) acc[j] = 0.0f;

            // tensorwise / rowwise scales; a warp's column scales wait in its part of the (otherwise unused) ring, fetched
            // before the tile's products are awaited: 128 loads per thread at the end of the tile made the
            // rowwise 8192^3 18 % slower than the tensorwise one
            float *my_cols = &ctl->scale_ring[(warp - 4) * kWgCols];
            float sa       = 1.0f;
            if constexpr (SCALE == kScaleTensor) sa = args.a_scale[0] * args.b_scale[0];
            if constexpr (SCALE == kScaleRow) {
                sa = args.a_scale[(int64_t) min(row, t.m_end - 1) * args.as_m];
                const float *bs = args.b_scale + (int64_t) gb * args.bs_g;
                __syncwarp(); // the previous tile's scales have been read
#pragma unroll
                for (int i = 0; i < kWgCols / 32; ++i)
                    my_cols[i * 32 + lane] = bs[(int64_t) min(col0 + i * 32 + lane, args.N - 1) * args.bs_n];
                __syncwarp();
            }

            // 1-D x 2-D block scales: each thread fetches its two scalars two contraction blocks
            // ahead of their use
            const float *a_sp = nullptr, *b_sp = nullptr;
            float sa0 = 0.f, sa1 = 0.f, sb0 = 0.f, sb1 = 0.f;
            if constexpr (SCALE == kScaleBlock2D) {
                a_sp = args.a_scale + (int64_t) min(row, t.m_end - 1) * args.as_m;
                b_sp = args.b_scale + (int64_t) gb * args.bs_g + (int64_t) min(col0 / 128, (args.N - 1) / 128) * args.bs_n;
                if (segs > 0) { sa0 = a_sp[0]; sb0 = b_sp[0]; }
                if (segs > 1) { sa1 = a_sp[args.as_k]; sb1 = b_sp[args.bs_k]; }
            }

            for (int sidx = 0; sidx < segs; ++sidx, ++acc_it) {
                const uint32_t buf = acc_it % kAccBufs;
                float s_row        = 1.0f;
                const float *cs    = nullptr;
                const int slot     = acc_it % kScaleSlots;
                if constexpr (SCALE == kScaleBlock1D) {
                    // this block's scales were copied into the ring by the loader warp, normally long ago
                    if (!mbar_wait(smem_u32(&ctl->sc_full[slot]), (acc_it / kScaleSlots) & 1)) { ok = false; break; }
                    const float *sl = &ctl->scale_ring[slot * kSlotFloats];
                    s_row           = sl[row_in_tile];
                    cs              = sl + 128 + wg * kWgCols;
                }
                if constexpr (SCALE == kScaleBlock2D) {
                    s_row = sa0 * sb0;
                    sa0   = sa1;
                    sb0   = sb1;
                    if (sidx + 2 < segs) {
                        sa1 = a_sp[(int64_t) (sidx + 2) * args.as_k];
                        sb1 = b_sp[(int64_t) (sidx + 2) * args.bs_k];
                    }
                }
                if (!mbar_wait(smem_u32(&ctl->tmem_full[buf]), (acc_it / kAccBufs) & 1)) { ok = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t) (quad * 32) << 16) + buf * BN + wg * kWgCols;
                const float2 s_row2  = make_float2(s_row, s_row);
                // two 32-column loads in flight; the second pair is issued while the first is consumed
                float v0[32], v1[32];
                tc_ld32(taddr, v0);
                tc_ld32(taddr + 32, v1);
                tc_wait_ld();
// packed fp32x2 arithmetic: half the issue slots of scalar FMA for the same IEEE results
#define PTB_PROMOTE(V, C)                                                                                      \
    _Pragma("unroll") for (int j = 0; j < 8; ++j) {                                      \
        float2 a0 = make_float2(acc[(C) * 32 + 4 * j], acc[(C) * 32 + 4 * j + 1]);                              \
        float2 a1 = make_float2(acc[(C) * 32 + 4 * j + 2], acc[(C) * 32 + 4 * j + 3]);                          \
        const float2 x0 = make_float2(V[4 * j], V[4 * j + 1]), x1 = make_float2(V[4 * j + 2], V[4 * j + 3]);     \
        if constexpr (SCALE == kScaleBlock2D) {                                                                 \
            a0 = __ffma2_rn(x0, s_row2, a0);                                                                    \
            a1 = __ffma2_rn(x1, s_row2, a1);                                                                    \
        } else if constexpr (SCALE == kScaleBlock1D) {                                                          \
            const float4 c4 = *reinterpret_cast<const float4 *>(cs + (C) * 32 + 4 * j);                          \
            a0 = __ffma2_rn(__fmul2_rn(x0, s_row2), make_float2(c4.x, c4.y), a0);                               \
            a1 = __ffma2_rn(__fmul2_rn(x1, s_row2), make_float2(c4.z, c4.w), a1);                               \
        } else {                                                                                                \
            a0 = x0;                                                                                            \
            a1 = x1;                                                                                            \
        }                                                                                                       \
        acc[(C) * 32 + 4 * j] = a0.x; acc[(C) * 32 + 4 * j + 1] = a0.y;                                         \
        acc[(C) * 32 + 4 * j + 2] = a1.x; acc[(C) * 32 + 4 * j + 3] = a1.y;                                     \
    }
                static_assert(kChunks == 4, "the promotion loop is written for four 32-column loads");
                PTB_PROMOTE(v0, 0)
                tc_ld32(taddr + 64, v0);
                PTB_PROMOTE(v1, 1)
                tc_ld32(taddr + 96, v1);
                tc_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { // buffer may be overwritten now
                    if constexpr (CTAS == 2) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(&ctl->tmem_empty[buf]), 0));
                    else mbar_arrive(smem_u32(&ctl->tmem_empty[buf]));
                }
                PTB_PROMOTE(v0, 2)
                PTB_PROMOTE(v1, 3)
#undef PTB_PROMOTE
                if constexpr (SCALE == kScaleBlock1D) {
                    __syncwarp(); // every lane has read its scales: the loader may refill the slot
                    if (lane == 0) mbar_arrive(smem_u32(&ctl->sc_empty[slot]));
                }
            }
            if (!ok) break;

            // ---- scale (tensorwise / rowwise), convert and store ---------------------------------
            if constexpr (SCALE == kScaleTensor) {
#pragma unroll
                for (int j = 0; j < kWgCols; ++j) acc[j] *= sa;
            }
            if constexpr (SCALE == kScaleRow) {
#pragma unroll
                for (int j = 0; j < kWgCols; j += 4) {
                    const float4 c4 = *reinterpret_cast<const float4 *>(my_cols + j);
                    acc[j] *= sa * c4.x; acc[j + 1] *= sa * c4.y; acc[j + 2] *= sa * c4.z; acc[j + 3] *= sa * c4.w;
                }
            }
            const int warp_row0 = t.m0 + quad * 32;
            if (tma_store && warp_row0 + 32 <= t.m_end) {
                // whole 32-row slab is inside the tile's valid rows: stage it (128-byte swizzled) and
                // let the copy engine write it; the tensor map clips columns past N
                if constexpr (sizeof(OutT) == 2) {
                    if (store_pending) {
                        if (lane == 0) tma_store_wait_read();
                        __syncwarp();
                    }
#pragma unroll
                    for (int j8 = 0; j8 < kWgCols / 8; ++j8) {
                        // one 16-byte shared store per lane: a quarter-warp writes eight different
                        // 16-byte columns of the swizzled slab (no bank conflict)
                        const uint32_t dst = stage_u32 + (j8 >> 3) * 4096 + lane * 128 + (((j8 & 7) ^ (lane & 7)) << 4);
                        st_shared_v4(dst, Pack8<OutT>::pack(&acc[j8 * 8]));
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        const int gc = (args.kind == kKindGroupedK) ? t.g : 0;
                        if (col0 < args.N) tma_store_3d(&args.tm_c, smem_u32(my_stage), col0, warp_row0, gc);
                        if (col0 + 64 < args.N) tma_store_3d(&args.tm_c, smem_u32(my_stage + 4096), col0 + 64, warp_row0, gc);
                        tma_store_commit();
                    }
                    store_pending = true;
                }
            } else if (row < t.m_end) {
                OutT *crow = cbase + (int64_t) t.g * args.c_group_stride + (int64_t) row * args.ldc;
#pragma unroll
                for (int j8 = 0; j8 < kWgCols / 8; ++j8) {
                    const int c = col0 + j8 * 8;
                    if (c >= args.N) continue;
                    if (vec_store && c + 8 <= args.N) {
                        Pack8<OutT>::store(crow + c, &acc[j8 * 8]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (c + j < args.N) crow[c + j] = from_f32<OutT>(acc[j8 * 8 + j]);
                    }
                }
            }
        }
        if (store_pending && lane == 0) tma_store_wait_all();
        if (!ok && lane == 0) atomicExch(&g_gemm_status, 3);
    }

    // ---- teardown -----------------------------------------------------------------------------------
    tc_fence_before();
    __syncthreads();
    // neither CTA of a pair leaves while the other may still signal its barriers or read its operands
    if constexpr (CTAS == 2) cluster_sync();
    if (warp == 2) {
        tc_fence_after();
        if constexpr (CTAS == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

// One warp waits on a barrier that nothing ever arrives on.  It exercises exactly the bounded wait the
// GEMM roles use: the wait gives up after its limit, the kernel records a status code and returns
// normally, and the context stays usable.
__global__ void __launch_bounds__(32) wait_selftest_kernel() {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    const bool ok = mbar_wait(smem_u32(&bar), 0);
    if (!ok && threadIdx.x == 0) atomicExch(&g_gemm_status, 9);
}

// ---- host side -------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int get_encode_fn(EncodeTiledFn *out) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetDriverEntryPoint(cuTensorMapEncodeTiled)");
        if (qres != cudaDriverEntryPointSuccess || !p)
            return fail(PTB_ERR_DRIVER, "cuTensorMapEncodeTiled is not available in this driver");
        fn = (EncodeTiledFn) p;
    }
    *out = fn;
    return 0;
}

// 3-D byte tensor {d0 (contiguous), d1, d2} with a {128, box1, 1} box and 128-byte swizzle.
int make_map(CUtensorMap *tm, const void *base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t pitch1,
             uint64_t pitch2, uint32_t box1) {
    EncodeTiledFn fn;
    int rc = get_encode_fn(&fn);
    if (rc) return rc;
    PTB_REQUIRE(aligned16(base), PTB_ERR_ALIGN, "GEMM operand base address is not 16-byte aligned");
    PTB_REQUIRE(pitch1 % 16 == 0 && pitch2 % 16 == 0, PTB_ERR_ALIGN,
                "GEMM operand leading dimension (%llu bytes) is not a multiple of 16", (unsigned long long) pitch1);
    cuuint64_t dims[3]    = {d0, d1 ? d1 : 1, d2 ? d2 : 1};
    cuuint64_t strides[2] = {pitch1, pitch2};
    cuuint32_t box[3]     = {128, box1, 1};
    cuuint32_t estr[3]    = {1, 1, 1};
    CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    PTB_REQUIRE(r == CUDA_SUCCESS, PTB_ERR_DRIVER, "cuTensorMapEncodeTiled failed with CUresult %d", (int) r);
    return 0;
}

// Output map for the TMA-store epilogue: 16-bit elements, {64, 32, 1} boxes, 128-byte swizzle.
// Returns 0 and sets *ok = 1 when the layout qualifies; otherwise the kernel stores directly.
int make_c_map(CUtensorMap *tm, int *ok, void *c, int out_dtype, uint64_t cols, uint64_t rows, uint64_t groups,
               uint64_t ldc, uint64_t group_stride) {
    *ok = 0;
    if (out_dtype != PTB_BF16 && out_dtype != PTB_F16) return 0;
    if (!aligned16(c) || (ldc * 2) % 16 != 0 || (group_stride * 2) % 16 != 0) return 0;
    EncodeTiledFn fn;
    int rc = get_encode_fn(&fn);
    if (rc) return rc;
    cuuint64_t dims[3]    = {cols, rows ? rows : 1, groups ? groups : 1};
    cuuint64_t strides[2] = {ldc * 2, (group_stride ? group_stride : ldc * (rows ? rows : 1)) * 2};
    cuuint32_t box[3]     = {64, 32, 1};
    cuuint32_t estr[3]    = {1, 1, 1};
    CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, c, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    PTB_REQUIRE(r == CUDA_SUCCESS, PTB_ERR_DRIVER, "cuTensorMapEncodeTiled (output) failed with CUresult %d", (int) r);
    *ok = 1;
    return 0;
}

uint32_t make_idesc(int a_dtype, int b_dtype, int a_mn, int b_mn, int BN, int ctas = 1) {
    uint32_t d = 0;
    d |= 1u << 4;                                    // D format fp32
    d |= (a_dtype == PTB_E5M2 ? 1u : 0u) << 7;       // A format
    d |= (b_dtype == PTB_E5M2 ? 1u : 0u) << 10;      // B format
    d |= (uint32_t) (a_mn ? 1 : 0) << 15;            // A major
    d |= (uint32_t) (b_mn ? 1 : 0) << 16;            // B major
    d |= (uint32_t) (BN >> 3) << 17;                 // N
    d |= (uint32_t) (ctas * BM >> 4) << 24;          // M
    return d;
}

// Block-scaled (MX) descriptor: no accumulator-format field; bits 4-5 and 29-30 select the scale byte
// of B and A (filled in per instruction), bit 23 says the scales are E8M0.
uint32_t make_idesc_mx(int a_dtype, int b_dtype, int BN) {
    uint32_t d = 0;
    d |= (a_dtype == PTB_E5M2 ? 1u : 0u) << 7;       // A format
    d |= (b_dtype == PTB_E5M2 ? 1u : 0u) << 10;      // B format
    d |= (uint32_t) (BN >> 3) << 17;                 // N
    d |= 1u << 23;                                   // scale format E8M0
    d |= (uint32_t) (BM >> 4) << 24;                 // M
    return d;
}

template <int BN, int DEEP, int CTAS> constexpr size_t smem_bytes() {
    using G_ = Geo<BN, DEEP, CTAS>;
    return 1024 + (size_t) G_::kStages * G_::kStageBytes + G_::kCStageBytes + sizeof(SharedCtl);
}
static_assert(smem_bytes<256, 0, 1>() <= 232448 && smem_bytes<256, 1, 1>() <= 232448 && smem_bytes<256, 0, 2>() <= 232448,
              "shared memory budget of one CTA exceeded");

template <int SCALE, typename OutT, int BN, int DEEP, int CTAS> int launch_bn(const GemmArgs &args, int grid, cudaStream_t st) {
    static bool configured[64] = {}; // per device; the attribute set is idempotent, a race only repeats it
    constexpr size_t kSmemBytes = smem_bytes<BN, DEEP, CTAS>();
    auto kfn = fp8_gemm_kernel<SCALE, OutT, BN, DEEP, CTAS>;
    int dev  = 0;
    PTB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        PTB_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kSmemBytes));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    PTB_CUDA((launch_after(kfn, dim3((unsigned) (CTAS == 2 ? grid & ~1 : grid)), Geo<BN, DEEP, CTAS>::kThreads, kSmemBytes, st, CTAS, args)));
    PTB_LAUNCH_CHECK("fp8_gemm_kernel");
    return 0;
}

template <int SCALE, typename OutT> int launch_one(const GemmArgs &args, int grid, cudaStream_t st) {
    constexpr bool kCanDeep = SCALE == kScaleTensor || SCALE == kScaleRow;
    if constexpr (kCanDeep) {
        if (args.ctas == 2) return launch_bn<SCALE, OutT, 256, 0, 2>(args, grid, st);
        if (args.deep) return launch_bn<SCALE, OutT, 256, 1, 1>(args, grid, st);
    }
    return launch_bn<SCALE, OutT, 256, 0, 1>(args, grid, st);
}

template <int SCALE> int launch_scale(const GemmArgs &args, int out_dtype, int grid, cudaStream_t st) {
    switch (out_dtype) {
    case PTB_BF16: return launch_one<SCALE, __nv_bfloat16>(args, grid, st);
    case PTB_F16: return launch_one<SCALE, __half>(args, grid, st);
    case PTB_F32: return launch_one<SCALE, float>(args, grid, st);
    default: return fail(PTB_ERR_ARG, "GEMM output dtype %d is not supported", out_dtype);
    }
}

// CTAs of a persistent launch: one per SM, or the caller's cap
int persistent_grid(int num_sms, int *grid) {
    int dev = 0, sms = 0;
    PTB_CUDA(cudaGetDevice(&dev));
    PTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    *grid = (num_sms > 0 && num_sms < sms) ? num_sms : sms;
    return 0;
}

constexpr int kTileN = 256;

// CTAs per tile.  Only tensorwise and rowwise scales run in pairs: with block scales the promotion warps set the pace
// and a second CTA's hand-shakes slow them (8192^3 NT, 128 x 128 weight blocks: 0.54 ms alone, 0.66 in pairs).  A contraction
// block of the one-CTA tile takes 855 clocks (48 KiB in and 48 KiB out of a 128 B/clock shared memory), of the
// pair's 730, so per SM a wave of pairs counts 6 / 7 of a wave of single tiles; where the 256-row tiles' padding or
// the last wave costs more than that, tiles stay single.  8192^3: tensorwise 424 -> 404 us, rowwise 498 -> 462 us.
int dense_ctas(int mode, int64_t M, int64_t N, int grid) {
    if ((mode != kScaleTensor && mode != kScaleRow) || grid < 2) return 1;
    const int64_t tn = cdiv<int64_t>(N, kTileN);
    return cdiv<int64_t>(cdiv<int64_t>(M, 2 * BM) * tn, grid / 2) * 6 <= cdiv<int64_t>(cdiv<int64_t>(M, BM) * tn, grid) * 7 ? 2 : 1;
}
// Row groups: how many rows each group has is known on the device only.  With uneven groups of 256 rows on average the
// 256-row tiles' padding eats the gain (log-normal loads: 317 single tiles against 2 x 198); from 384 on it does not.
int grouped_ctas(int mode, int64_t rows, int64_t G, int grid) {
    return (mode == kScaleTensor || mode == kScaleRow) && grid >= 2 && rows >= 384 * G ? 2 : 1;
}

int launch_gemm(GemmArgs &args, int scale_mode, int out_dtype, int grid, cudaStream_t st) {
    // Tensorwise / rowwise scales keep the whole K loop in TMEM, so the epilogue is rare: spend the
    // staging buffer on a fourth pipeline stage instead (measured +8 % on 8192^3).
    // (A pair's stages are smaller: it has four beside the staging buffer.)
    args.deep = (scale_mode == kScaleTensor || scale_mode == kScaleRow) && args.kind == kKindDense && args.ctas == 1 ? 1 : 0;
    switch (scale_mode) {
    case kScaleTensor: return launch_scale<kScaleTensor>(args, out_dtype, grid, st);
    case kScaleRow: return launch_scale<kScaleRow>(args, out_dtype, grid, st);
    case kScaleBlock2D: return launch_scale<kScaleBlock2D>(args, out_dtype, grid, st);
    case kScaleBlock1D: return launch_scale<kScaleBlock1D>(args, out_dtype, grid, st);
    case kScaleMX: return launch_scale<kScaleMX>(args, out_dtype, grid, st);
    default: return fail(PTB_ERR_ARG, "unknown scale mode %d", scale_mode);
    }
}

// the fields every entry point derives from the number of CTAs per tile
void set_tile(GemmArgs &g, int ctas) {
    g.ctas = ctas;
    g.bm   = ctas * BM;
    g.bn   = kTileN;
}

int scale_mode_of(int granularity, int b_block_2d, int *mode) {
    switch (granularity) {
    case PTB_TENSORWISE: *mode = kScaleTensor; return 0;
    case PTB_ROWWISE: *mode = kScaleRow; return 0;
    case PTB_BLOCKWISE: *mode = b_block_2d ? kScaleBlock2D : kScaleBlock1D; return 0;
    default: return fail(PTB_ERR_ARG, "unknown granularity %d", granularity);
    }
}

} // namespace
} // namespace ptb

#include "ptb_gemm_skinny.cuh"
#include "ptb_gemm_wgrad.cuh"

// Build-time switch for A/B measurements of the two wgrad kernels (1: paired-tile kernel where it applies).
#ifndef PTB_WGRAD_PAIR
#define PTB_WGRAD_PAIR 1
#endif

using namespace ptb;

extern "C" {
#pragma GCC visibility push(default)

int ptb_gemm_wait_selftest(ptb_stream_t stream) {
    wait_selftest_kernel<<<1, 32, 0, (cudaStream_t) stream>>>();
    PTB_LAUNCH_CHECK("wait_selftest_kernel");
    return 0;
}

int ptb_gemm_status(int *status, int reset) {
    PTB_REQUIRE(status, PTB_ERR_ARG, "gemm_status: null pointer");
    PTB_CUDA(cudaMemcpyFromSymbol(status, g_gemm_status, sizeof(int)));
    if (reset) {
        int zero = 0;
        PTB_CUDA(cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(int)));
    }
    return 0;
}

int ptb_gemm_fp8(const void *a, int a_dtype, int trans_a, int64_t lda, const void *b, int b_dtype, int trans_b,
                 int64_t ldb, void *c, int c_dtype, int64_t ldc, int64_t M, int64_t N, int64_t K, int granularity,
                 const float *a_scale, int64_t a_scale_stride_m, int64_t a_scale_stride_k, const float *b_scale,
                 int64_t b_scale_stride_n, int64_t b_scale_stride_k, int b_block_2d, int num_sms,
                 ptb_stream_t stream) {
    PTB_REQUIRE(M >= 0 && N >= 0 && K > 0, PTB_ERR_ARG, "gemm_fp8: bad shape M=%lld N=%lld K=%lld", (long long) M,
                (long long) N, (long long) K);
    if (M == 0 || N == 0) return 0;
    PTB_REQUIRE(a && b && c && a_scale && b_scale, PTB_ERR_ARG, "gemm_fp8: null pointer");
    PTB_REQUIRE(is_fp8(a_dtype) && is_fp8(b_dtype), PTB_ERR_ARG, "gemm_fp8: operands must be FP8");
    PTB_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), PTB_ERR_TOO_LARGE, "gemm_fp8: dimension too large");
    int mode;
    int rc = scale_mode_of(granularity, b_block_2d, &mode);
    if (rc) return rc;
    GemmArgs g{};
    const int BN = kTileN;
    int grid = 0;
    rc       = persistent_grid(num_sms, &grid);
    if (rc) return rc;
    g.kind = kKindDense;
    g.M = (int) M; g.N = (int) N; g.K = (int) K; g.G = 1;
    g.c = c; g.ldc = ldc; g.c_group_stride = 0;
    g.a_scale = a_scale; g.as_m = a_scale_stride_m; g.as_k = a_scale_stride_k;
    g.b_scale = b_scale; g.bs_g = 0; g.bs_n = b_scale_stride_n; g.bs_k = b_scale_stride_k;
    if (const int tn = skinny_rows(mode, M, 0, N, !trans_a && trans_b, grid))
        return launch_skinny(g, mode, tn, a, a_dtype, lda, b, b_dtype, ldb, 1, c_dtype, grid, (cudaStream_t) stream);
    const int ctas = dense_ctas(mode, M, N, grid);
    set_tile(g, ctas);
    // A: [M,K] K-major, or [K,M] (trans_a) MN-major
    if (!trans_a) rc = make_map(&g.tm_a, a, (uint64_t) K, (uint64_t) M, 1, (uint64_t) lda, (uint64_t) lda * M, BM);
    else          rc = make_map(&g.tm_a, a, (uint64_t) M, (uint64_t) K, 1, (uint64_t) lda, (uint64_t) lda * K, BK);
    if (rc) return rc;
    // B: [N,K] (trans_b) K-major, or [K,N] MN-major
    if (trans_b) rc = make_map(&g.tm_b, b, (uint64_t) K, (uint64_t) N, 1, (uint64_t) ldb, (uint64_t) ldb * N, BN / ctas);
    else         rc = make_map(&g.tm_b, b, (uint64_t) N, (uint64_t) K, 1, (uint64_t) ldb, (uint64_t) ldb * K, BK);
    if (rc) return rc;
    g.a_mn = trans_a ? 1 : 0; g.b_mn = trans_b ? 0 : 1;
    g.idesc = make_idesc(a_dtype, b_dtype, g.a_mn, g.b_mn, BN, ctas);
    g.tiles_n = (int) cdiv<int64_t>(N, BN);
    rc = make_c_map(&g.tm_c, &g.use_tma_store, c, c_dtype, (uint64_t) N, (uint64_t) M, 1, (uint64_t) ldc, 0);
    if (rc) return rc;
    return launch_gemm(g, mode, c_dtype, grid, (cudaStream_t) stream);
}

int ptb_gemm_mxfp8(const void *a, int a_dtype, int64_t lda, const void *a_sf, int64_t a_sf_ld, const void *b, int b_dtype,
                   int64_t ldb, const void *b_sf, int64_t b_sf_ld, void *c, int c_dtype, int64_t ldc, int64_t M, int64_t N,
                   int64_t K, int num_sms, ptb_stream_t stream) {
    PTB_REQUIRE(M >= 0 && N >= 0 && K > 0, PTB_ERR_ARG, "gemm_mxfp8: bad shape M=%lld N=%lld K=%lld", (long long) M,
                (long long) N, (long long) K);
    if (M == 0 || N == 0) return 0;
    PTB_REQUIRE(a && b && c && a_sf && b_sf, PTB_ERR_ARG, "gemm_mxfp8: null pointer");
    PTB_REQUIRE(is_fp8(a_dtype) && is_fp8(b_dtype), PTB_ERR_ARG, "gemm_mxfp8: operands must be FP8");
    PTB_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), PTB_ERR_TOO_LARGE, "gemm_mxfp8: dimension too large");
    PTB_REQUIRE(K % BK == 0, PTB_ERR_ARG, "gemm_mxfp8: the (padded) contraction extent %lld must be a multiple of 128", (long long) K);
    PTB_REQUIRE(a_sf_ld >= K / 32 && b_sf_ld >= K / 32 && a_sf_ld % 4 == 0 && b_sf_ld % 4 == 0 &&
                    (reinterpret_cast<uintptr_t>(a_sf) & 3u) == 0 && (reinterpret_cast<uintptr_t>(b_sf) & 3u) == 0,
                PTB_ERR_ALIGN, "gemm_mxfp8: scale rows must hold K/32 bytes, be 4-byte aligned and a multiple of 4 bytes apart");
    GemmArgs g{};
    const int BN = kTileN;
    set_tile(g, 1);
    int rc = make_map(&g.tm_a, a, (uint64_t) K, (uint64_t) M, 1, (uint64_t) lda, (uint64_t) lda * M, BM);
    if (rc) return rc;
    rc = make_map(&g.tm_b, b, (uint64_t) K, (uint64_t) N, 1, (uint64_t) ldb, (uint64_t) ldb * N, BN);
    if (rc) return rc;
    g.kind = kKindDense; g.a_mn = 0; g.b_mn = 0;
    g.idesc = make_idesc_mx(a_dtype, b_dtype, BN);
    g.M = (int) M; g.N = (int) N; g.K = (int) K; g.G = 1;
    g.tiles_n = (int) cdiv<int64_t>(N, BN);
    g.c = c; g.ldc = ldc; g.c_group_stride = 0;
    rc = make_c_map(&g.tm_c, &g.use_tma_store, c, c_dtype, (uint64_t) N, (uint64_t) M, 1, (uint64_t) ldc, 0);
    if (rc) return rc;
    g.a_sf = (const uint8_t *) a_sf; g.a_sf_ld = a_sf_ld; g.b_sf = (const uint8_t *) b_sf; g.b_sf_ld = b_sf_ld;
    int grid = 0;
    rc       = persistent_grid(num_sms, &grid);
    if (rc) return rc;
    return launch_gemm(g, kScaleMX, c_dtype, grid, (cudaStream_t) stream);
}

int ptb_grouped_gemm_mxfp8(const void *a, int a_dtype, int64_t lda, const void *a_sf, int64_t a_sf_ld, const void *b,
                           int b_dtype, const void *b_sf, void *out, int out_dtype, int64_t ldc, const int64_t *group_offs,
                           int64_t G, int64_t M_total, int64_t N, int64_t K, int num_sms, ptb_stream_t stream) {
    PTB_REQUIRE(G >= 0 && M_total >= 0 && N >= 0 && K > 0, PTB_ERR_ARG, "grouped_gemm_mxfp8: bad shape");
    if (M_total == 0 || N == 0) return 0;
    PTB_REQUIRE(G > 0 && G <= kMaxGroups, PTB_ERR_TOO_LARGE, "grouped_gemm_mxfp8: 1 to %d groups", kMaxGroups);
    PTB_REQUIRE(a && b && out && group_offs && a_sf && b_sf, PTB_ERR_ARG, "grouped_gemm_mxfp8: null pointer");
    PTB_REQUIRE(is_fp8(a_dtype) && is_fp8(b_dtype), PTB_ERR_ARG, "grouped_gemm_mxfp8: operands must be FP8");
    PTB_REQUIRE(M_total < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31) && G * N < (1ll << 31), PTB_ERR_TOO_LARGE,
                "grouped_gemm_mxfp8: dimension too large");
    PTB_REQUIRE(K % BK == 0, PTB_ERR_ARG, "grouped_gemm_mxfp8: the (padded) contraction extent %lld must be a multiple of 128",
                (long long) K);
    PTB_REQUIRE(a_sf_ld >= K / 32 && a_sf_ld % 4 == 0 && (reinterpret_cast<uintptr_t>(a_sf) & 3u) == 0 &&
                    (reinterpret_cast<uintptr_t>(b_sf) & 3u) == 0,
                PTB_ERR_ALIGN, "grouped_gemm_mxfp8: scale rows must hold K/32 bytes, be 4-byte aligned and a multiple of 4 apart");
    GemmArgs g{};
    const int BN = kTileN;
    set_tile(g, 1);
    int rc = make_map(&g.tm_a, a, (uint64_t) K, (uint64_t) M_total, 1, (uint64_t) lda, (uint64_t) lda * M_total, BM);
    if (rc) return rc;
    rc = make_map(&g.tm_b, b, (uint64_t) K, (uint64_t) N, (uint64_t) G, (uint64_t) K, (uint64_t) K * N, BN);
    if (rc) return rc;
    g.kind = kKindGroupedRows; g.a_mn = 0; g.b_mn = 0;
    g.idesc = make_idesc_mx(a_dtype, b_dtype, BN);
    g.M = (int) M_total; g.N = (int) N; g.K = (int) K; g.G = (int) G;
    g.tiles_n = (int) cdiv<int64_t>(N, BN);
    g.group_offs = group_offs;
    g.c = out; g.ldc = ldc; g.c_group_stride = 0;
    rc = make_c_map(&g.tm_c, &g.use_tma_store, out, out_dtype, (uint64_t) N, (uint64_t) M_total, 1, (uint64_t) ldc, 0);
    if (rc) return rc;
    g.a_sf = (const uint8_t *) a_sf; g.a_sf_ld = a_sf_ld; g.b_sf = (const uint8_t *) b_sf; g.b_sf_ld = K / 32;
    int grid = 0;
    rc       = persistent_grid(num_sms, &grid);
    if (rc) return rc;
    return launch_gemm(g, kScaleMX, out_dtype, grid, (cudaStream_t) stream);
}

int ptb_grouped_gemm_mxfp8_variable_k(const void *lhs, int lhs_dtype, int64_t ld_lhs, const void *lhs_sf, int64_t lhs_sf_ld,
                                      const void *rhs, int rhs_dtype, int64_t ld_rhs, const void *rhs_sf, int64_t rhs_sf_ld,
                                      void *out, int out_dtype, const int64_t *group_offs_padded, int64_t G, int64_t rows_padded,
                                      int64_t OUT_M, int64_t OUT_N, int num_sms, ptb_stream_t stream) {
    PTB_REQUIRE(G >= 0 && rows_padded >= 0 && OUT_M >= 0 && OUT_N >= 0, PTB_ERR_ARG, "grouped_gemm_mxfp8_variable_k: bad shape");
    if (G == 0 || OUT_M == 0 || OUT_N == 0) return 0;
    PTB_REQUIRE(lhs && rhs && out && group_offs_padded && lhs_sf && rhs_sf, PTB_ERR_ARG,
                "grouped_gemm_mxfp8_variable_k: null pointer");
    PTB_REQUIRE(is_fp8(lhs_dtype) && is_fp8(rhs_dtype), PTB_ERR_ARG, "grouped_gemm_mxfp8_variable_k: operands must be FP8");
    PTB_REQUIRE(G <= kMaxGroups, PTB_ERR_TOO_LARGE, "grouped_gemm_mxfp8_variable_k: at most %d groups", kMaxGroups);
    PTB_REQUIRE(rows_padded % BK == 0, PTB_ERR_ARG, "grouped_gemm_mxfp8_variable_k: padded rows must be a multiple of 128");
    PTB_REQUIRE(rows_padded < (1ll << 31) && OUT_M < (1ll << 31) && OUT_N < (1ll << 31) &&
                    G * cdiv<int64_t>(OUT_M, BM) * cdiv<int64_t>(OUT_N, 128) < (1ll << 31),
                PTB_ERR_TOO_LARGE, "grouped_gemm_mxfp8_variable_k: problem too large");
    PTB_REQUIRE(lhs_sf_ld >= rows_padded / 32 && rhs_sf_ld >= rows_padded / 32 && lhs_sf_ld % 4 == 0 && rhs_sf_ld % 4 == 0 &&
                    (reinterpret_cast<uintptr_t>(lhs_sf) & 3u) == 0 && (reinterpret_cast<uintptr_t>(rhs_sf) & 3u) == 0,
                PTB_ERR_ALIGN, "grouped_gemm_mxfp8_variable_k: scale rows must be 4-byte aligned and a multiple of 4 apart");
    GemmArgs g{};
    const int BN = kTileN;
    set_tile(g, 1);
    const uint64_t r = rows_padded > 0 ? (uint64_t) rows_padded : 1;
    // both operands are transposed copies: [OUT_M, rows] and [OUT_N, rows], contraction axis contiguous
    int rc = make_map(&g.tm_a, lhs, r, (uint64_t) OUT_M, 1, (uint64_t) ld_lhs, (uint64_t) ld_lhs * OUT_M, BM);
    if (rc) return rc;
    rc = make_map(&g.tm_b, rhs, r, (uint64_t) OUT_N, 1, (uint64_t) ld_rhs, (uint64_t) ld_rhs * OUT_N, BN);
    if (rc) return rc;
    g.kind = kKindGroupedK; g.a_mn = 0; g.b_mn = 0;
    g.idesc = make_idesc_mx(lhs_dtype, rhs_dtype, BN);
    g.M = (int) OUT_M; g.N = (int) OUT_N; g.K = (int) rows_padded; g.G = (int) G;
    g.tiles_n = (int) cdiv<int64_t>(OUT_N, BN);
    g.group_offs = group_offs_padded;
    g.c = out; g.ldc = OUT_N; g.c_group_stride = OUT_M * OUT_N;
    rc = make_c_map(&g.tm_c, &g.use_tma_store, out, out_dtype, (uint64_t) OUT_N, (uint64_t) OUT_M, (uint64_t) G,
                    (uint64_t) OUT_N, (uint64_t) (OUT_M * OUT_N));
    if (rc) return rc;
    g.a_sf = (const uint8_t *) lhs_sf; g.a_sf_ld = lhs_sf_ld; g.b_sf = (const uint8_t *) rhs_sf; g.b_sf_ld = rhs_sf_ld;
    int grid = 0;
    rc       = persistent_grid(num_sms, &grid);
    if (rc) return rc;
    return launch_gemm(g, kScaleMX, out_dtype, grid, (cudaStream_t) stream);
}

int ptb_grouped_gemm_fp8(const void *a, int a_dtype, int64_t lda, const void *b, int b_dtype, int trans_b, void *out,
                         int out_dtype, int64_t ldc, const int64_t *group_offs, int64_t G, int64_t M_total, int64_t N,
                         int64_t K, int granularity, const float *a_scale, int64_t a_scale_stride_m,
                         int64_t a_scale_stride_k, const float *b_scale, int64_t b_scale_stride_g,
                         int64_t b_scale_stride_n, int64_t b_scale_stride_k, int num_sms, ptb_stream_t stream) {
    PTB_REQUIRE(G >= 0 && M_total >= 0 && N >= 0 && K > 0, PTB_ERR_ARG, "grouped_gemm_fp8: bad shape");
    if (M_total == 0 || N == 0) return 0;
    PTB_REQUIRE(G > 0, PTB_ERR_ARG, "grouped_gemm_fp8: no groups");
    PTB_REQUIRE(G <= kMaxGroups, PTB_ERR_TOO_LARGE, "grouped_gemm_fp8: at most %d groups", kMaxGroups);
    PTB_REQUIRE(a && b && out && group_offs && a_scale && b_scale, PTB_ERR_ARG, "grouped_gemm_fp8: null pointer");
    PTB_REQUIRE(is_fp8(a_dtype) && is_fp8(b_dtype), PTB_ERR_ARG, "grouped_gemm_fp8: operands must be FP8");
    PTB_REQUIRE(M_total < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), PTB_ERR_TOO_LARGE,
                "grouped_gemm_fp8: dimension too large");
    int mode;
    int rc = scale_mode_of(granularity, 1, &mode);
    if (rc) return rc;
    GemmArgs g{};
    const int BN = kTileN;
    int grid = 0;
    rc       = persistent_grid(num_sms, &grid);
    if (rc) return rc;
    g.kind = kKindGroupedRows;
    g.M = (int) M_total; g.N = (int) N; g.K = (int) K; g.G = (int) G;
    g.group_offs = group_offs;
    g.c = out; g.ldc = ldc; g.c_group_stride = 0;
    g.a_scale = a_scale; g.as_m = a_scale_stride_m; g.as_k = a_scale_stride_k;
    g.b_scale = b_scale; g.bs_g = b_scale_stride_g; g.bs_n = b_scale_stride_n; g.bs_k = b_scale_stride_k;
    if (const int tn = skinny_rows(mode, M_total, G, N, trans_b != 0, grid))
        return launch_skinny(g, mode, tn, a, a_dtype, lda, b, b_dtype, K, (uint64_t) G, out_dtype, grid, (cudaStream_t) stream);
    const int ctas = grouped_ctas(mode, M_total, G, grid);
    set_tile(g, ctas);
    rc = make_map(&g.tm_a, a, (uint64_t) K, (uint64_t) M_total, 1, (uint64_t) lda, (uint64_t) lda * M_total, BM);
    if (rc) return rc;
    if (trans_b) rc = make_map(&g.tm_b, b, (uint64_t) K, (uint64_t) N, (uint64_t) G, (uint64_t) K, (uint64_t) K * N, BN / ctas);
    else         rc = make_map(&g.tm_b, b, (uint64_t) N, (uint64_t) K, (uint64_t) G, (uint64_t) N, (uint64_t) K * N, BK);
    if (rc) return rc;
    g.a_mn = 0; g.b_mn = trans_b ? 0 : 1;
    g.idesc = make_idesc(a_dtype, b_dtype, g.a_mn, g.b_mn, BN, ctas);
    g.tiles_n = (int) cdiv<int64_t>(N, BN);
    rc = make_c_map(&g.tm_c, &g.use_tma_store, out, out_dtype, (uint64_t) N, (uint64_t) M_total, 1, (uint64_t) ldc, 0);
    if (rc) return rc;
    return launch_gemm(g, mode, out_dtype, grid, (cudaStream_t) stream);
}

int ptb_grouped_gemm_fp8_variable_k(const void *lhs, int lhs_dtype, int64_t ld_lhs, const void *rhs, int rhs_dtype,
                                    int64_t ld_rhs, void *out, int out_dtype, const int64_t *group_offs, int64_t G,
                                    int64_t rows, int64_t OUT_M, int64_t OUT_N, int granularity,
                                    const float *lhs_scale, const float *rhs_scale, int num_sms,
                                    ptb_stream_t stream) {
    PTB_REQUIRE(G >= 0 && rows >= 0 && OUT_M >= 0 && OUT_N >= 0, PTB_ERR_ARG, "grouped_gemm_fp8_variable_k: bad shape");
    if (G == 0 || OUT_M == 0 || OUT_N == 0) return 0;
    int mode;
    int rc = scale_mode_of(granularity, 0, &mode);
    if (rc) return rc;
    PTB_REQUIRE(lhs && rhs && out && group_offs && lhs_scale && rhs_scale, PTB_ERR_ARG,
                "grouped_gemm_fp8_variable_k: null pointer");
    PTB_REQUIRE(is_fp8(lhs_dtype) && is_fp8(rhs_dtype), PTB_ERR_ARG, "grouped_gemm_fp8_variable_k: operands must be FP8");
    PTB_REQUIRE(G <= kMaxGroups, PTB_ERR_TOO_LARGE, "grouped_gemm_fp8_variable_k: at most %d groups", kMaxGroups);
    PTB_REQUIRE(rows < (1ll << 31) && OUT_M < (1ll << 31) && OUT_N < (1ll << 31) &&
                    G * cdiv<int64_t>(OUT_M, BM) * cdiv<int64_t>(OUT_N, 128) < (1ll << 31),
                PTB_ERR_TOO_LARGE, "grouped_gemm_fp8_variable_k: problem too large");
    GemmArgs g{};
    const int BN = kTileN;
    int grid = 0;
    rc       = persistent_grid(num_sms, &grid);
    if (rc) return rc;
    const int ctas = (mode == kScaleTensor || mode == kScaleRow) && OUT_M > BM && grid >= 2 ? 2 : 1;
    set_tile(g, ctas);
    const uint64_t r = rows > 0 ? (uint64_t) rows : 1;
    rc = make_map(&g.tm_a, lhs, (uint64_t) OUT_M, r, 1, (uint64_t) ld_lhs, (uint64_t) ld_lhs * r, BK);
    if (rc) return rc;
    rc = make_map(&g.tm_b, rhs, (uint64_t) OUT_N, r, 1, (uint64_t) ld_rhs, (uint64_t) ld_rhs * r, BK);
    if (rc) return rc;
    g.kind = kKindGroupedK; g.a_mn = 1; g.b_mn = 1;
    g.idesc = make_idesc(lhs_dtype, rhs_dtype, 1, 1, BN, ctas);
    g.M = (int) OUT_M; g.N = (int) OUT_N; g.K = (int) rows; g.G = (int) G;
    g.tiles_n = (int) cdiv<int64_t>(OUT_N, BN);
    g.group_offs = group_offs;
    g.c = out; g.ldc = OUT_N; g.c_group_stride = OUT_M * OUT_N;
    rc = make_c_map(&g.tm_c, &g.use_tma_store, out, out_dtype, (uint64_t) OUT_N, (uint64_t) OUT_M, (uint64_t) G,
                    (uint64_t) OUT_N, (uint64_t) (OUT_M * OUT_N));
    if (rc) return rc;
    g.a_scale = lhs_scale; g.as_m = 1; g.as_k = OUT_M;
    g.b_scale = rhs_scale; g.bs_g = 0; g.bs_n = 1; g.bs_k = OUT_N;
    if (PTB_WGRAD_PAIR && mode == kScaleBlock1D && OUT_M % 256 == 0 && OUT_N % 128 == 0 && g.use_tma_store &&
        (out_dtype == PTB_BF16 || out_dtype == PTB_F16) && aligned16(lhs_scale) && aligned16(rhs_scale)) {
        // blockwise wgrad on tile-aligned shapes: 256 x 128 paired tiles (see ptb_gemm_wgrad.cuh)
        g.bn = 128;
        g.idesc = make_idesc(lhs_dtype, rhs_dtype, 1, 1, 128);
        return out_dtype == PTB_BF16 ? launch_wgrad_pair<__nv_bfloat16>(g, grid, (cudaStream_t) stream)
                                     : launch_wgrad_pair<__half>(g, grid, (cudaStream_t) stream);
    }
    return launch_gemm(g, mode, out_dtype, grid, (cudaStream_t) stream);
}

#pragma GCC visibility pop
} // extern "C"
