// FP8 GEMM / grouped GEMM for few rows against a large K-major weight (decode): out[t, n] = sum_k a[t, k] * w[n, k].
// Included by ptb_gemm.cu; shares its barriers, tile walk and bounded waits.
//
// What bounds it is the weight, read once from HBM.  The 128 x 256 tile makes the few rows the 128-row side: it loads 128
// rows of `a` for the 8 or 32 that exist (half as many bytes again through L2 and shared memory), and 256 weight rows
// a tile leave SMs without work (N = 14336: 56 tiles for 148 SMs; 32 experts x 4096: 512 tiles, 3.5 waves).  Here the
// operands change places: 128 weight rows are the MMA's M side, TN = 32, 64 or 128 rows of `a` its N side, so twice the
// tiles, a stage of 16 KiB of weight plus TN x 128 bytes, and an accumulator of TN columns.  A product's terms and
// the order they are added in are the same, so the results are too.
// 32 x 14336 x 4096 tensorwise: 19 -> 15 us; 32 experts x 4096 x 7168 tensorwise, 256 rows: the whole call 186 -> 175 us.
//
// One persistent CTA per SM, 256 threads: warp 0 TMA producer, warp 1 MMA issuer, warp 2 owns tensor memory, warp 3 loads
// block scales, warps 4-7 read the accumulator (lane = weight row, registers = rows of `a`), scale and store: the 32
// lanes of a warp hold 32 neighbouring columns of one output row, a 64-byte run per store.
#pragma once

namespace ptb {
namespace {

template <int TN> struct SkinnyGeo {
    static constexpr int kWBytes     = 128 * BK;
    static constexpr int kStageBytes = kWBytes + TN * BK;
    static constexpr int kStages     = TN <= 64 ? 8 : 6;
    static constexpr int kAccBufs    = 4;
    static constexpr int kThreads    = 256;
    static_assert(kStages <= kMaxStages && kAccBufs * TN <= 512 && TN + 1 <= kSlotFloats, "out of shared or tensor memory");
    static constexpr size_t kSmem    = 1024 + (size_t) kStages * kStageBytes + sizeof(SharedCtl);
    static_assert(kSmem <= 232448, "shared memory budget of one CTA exceeded");
};

// args as for fp8_gemm_kernel with bm = TN (rows of a), bn = 128 (weight rows); tm_a has TN-row boxes, tm_b 128-row boxes
template <int SCALE, typename OutT, int TN>
__global__ void __launch_bounds__(SkinnyGeo<TN>::kThreads, 1) skinny_gemm_kernel(const __grid_constant__ GemmArgs args) {
    using G_ = SkinnyGeo<TN>;
    constexpr int kStages = G_::kStages, kStageBytes = G_::kStageBytes, kAccBufs = G_::kAccBufs;
    constexpr bool kPerBlock = SCALE == kScaleBlock2D;
    static_assert(SCALE == kScaleTensor || SCALE == kScaleRow || SCALE == kScaleBlock2D, "scale mode");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem  = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    SharedCtl *ctl = reinterpret_cast<SharedCtl *>(smem + kStages * kStageBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = smem_u32(smem);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&ctl->full[s]), 1);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
        }
        for (int b = 0; b < kAccBufs; ++b) {
            mbar_init(smem_u32(&ctl->tmem_full[b]), 1);
            mbar_init(smem_u32(&ctl->tmem_empty[b]), 4);
        }
        for (int b = 0; b < kScaleSlots; ++b) {
            mbar_init(smem_u32(&ctl->sc_full[b]), 32);
            mbar_init(smem_u32(&ctl->sc_empty[b]), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        ctl->sched_q   = (int) gridDim.x / args.tiles_n;
        ctl->sched_rem = (int) gridDim.x % args.tiles_n;
    }
    if (threadIdx.x == 64) {
        tma_prefetch_map(&args.tm_a);
        tma_prefetch_map(&args.tm_b);
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&ctl->tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    grid_dep_begin(); // everything above touches no global memory
    if (args.kind == kKindGroupedRows) {
        for (int g = threadIdx.x; g <= args.G; g += G_::kThreads) ctl->group_offs[g] = (int) args.group_offs[g];
        if (warp == 3) { // cumulative row tiles per group (G <= kMaxGroups, checked on the host)
            int run = 0;
            for (int base = 0; base < args.G; base += 32) {
                const int g = base + lane;
                int inc     = g < args.G ? (int) ((args.group_offs[g + 1] - args.group_offs[g] + TN - 1) / TN) : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int n = __shfl_up_sync(0xffffffffu, inc, o);
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
        ctl->total_tiles = (args.M + TN - 1) / TN * args.tiles_n;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;

    Schedule sched(args, ctl);
    Tile t;
    bool ok = true;
    if (warp == 0) {
        // ================= TMA producer =================
        if (lane == 0) {
            uint32_t it = 0;
            while (ok && sched.get(t)) {
                const int gb = args.kind == kKindGroupedRows ? t.g : 0;
                for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
                    const int s = it % kStages;
                    if (!mbar_wait(smem_u32(&ctl->empty[s]), ((it / kStages) & 1) ^ 1)) { ok = false; break; }
                    const uint32_t full = smem_u32(&ctl->full[s]), sw = smem_base + s * kStageBytes;
                    mbar_expect_tx(full, kStageBytes);
                    tma_load_3d(sw, &args.tm_b, full, kb * BK, t.n0, gb);
                    tma_load_3d(sw + G_::kWBytes, &args.tm_a, full, kb * BK, t.m0, 0);
                }
            }
            if (!ok) {
                atomicExch(&g_gemm_status, 1);
                // let the copies already issued land before the CTA releases its shared memory
                const uint32_t back = it < (uint32_t) kStages ? it : (uint32_t) kStages;
                for (uint32_t j = 1; j <= back; ++j) {
                    const uint32_t q = it - j;
                    mbar_wait(smem_u32(&ctl->full[q % kStages]), (q / kStages) & 1);
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer (whole warp walks, lane 0 issues) =================
        uint32_t it = 0, acc_it = 0;
        while (ok && sched.get(t)) {
            for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
                const int s = it % kStages;
                const bool new_acc = kPerBlock || kb == 0;
                const uint32_t buf = acc_it % kAccBufs;
                if (new_acc && !mbar_wait(smem_u32(&ctl->tmem_empty[buf]), ((acc_it / kAccBufs) & 1) ^ 1)) { ok = false; break; }
                if (!mbar_wait(smem_u32(&ctl->full[s]), (it / kStages) & 1)) { ok = false; break; }
                __syncwarp();
                tc_fence_after();
                const bool last = kPerBlock || kb == t.num_kb - 1;
                if (lane == 0) {
                    const uint32_t sw = smem_base + s * kStageBytes;
                    const uint64_t wd = make_smem_desc(sw, 0, 1024), xd = make_smem_desc(sw + G_::kWBytes, 0, 1024);
#pragma unroll
                    for (int j = 0; j < BK / 32; ++j)
                        tc_mma_f8<1>(tmem_base + buf * TN, wd + 2 * j, xd + 2 * j, args.idesc, (j > 0 || !new_acc) ? 1u : 0u);
                    tc_commit(smem_u32(&ctl->empty[s]));
                    if (last) tc_commit(smem_u32(&ctl->tmem_full[buf]));
                }
                if (last) ++acc_it;
            }
        }
        if (!ok && lane == 0) atomicExch(&g_gemm_status, 2);
    } else if (warp == 3) {
        // ================= block scales: per contraction block, one per row of a and one for the 128 weight rows =========
        if constexpr (kPerBlock) {
            uint32_t it = 0;
            while (ok && sched.get(t)) {
                const int gb       = args.kind == kKindGroupedRows ? t.g : 0;
                const float *b_src = args.b_scale + (int64_t) gb * args.bs_g + (int64_t) (t.n0 / 128) * args.bs_n;
                for (int kb = 0; kb < t.num_kb; ++kb, ++it) {
                    const int slot = it % kScaleSlots;
                    if (!mbar_wait(smem_u32(&ctl->sc_empty[slot]), ((it / kScaleSlots) & 1) ^ 1)) { ok = false; break; }
                    float *dst = &ctl->scale_ring[slot * kSlotFloats];
#pragma unroll
                    for (int i = 0; i < TN / 32; ++i) {
                        const int r = min(t.m0 + i * 32 + lane, t.m_end - 1); // rows past the group are never stored
                        cp_async_f32(dst + i * 32 + lane, args.a_scale + (int64_t) r * args.as_m + (int64_t) kb * args.as_k);
                    }
                    if (lane == 0) cp_async_f32(dst + TN, b_src + (int64_t) kb * args.bs_k);
                    cp_async_arrive_on(smem_u32(&ctl->sc_full[slot]));
                }
            }
            cp_async_wait_all();
            if (!ok && lane == 0) atomicExch(&g_gemm_status, 4);
        }
    } else if (warp >= 4) {
        // ================= accumulator -> output =================
        const int quad = warp & 3;
        OutT *cbase    = reinterpret_cast<OutT *>(args.c);
        if (args.kind == kKindGroupedRows) {
            // zero the rows past the last group (the output is allocated for M rows)
            const int64_t first = args.group_offs[args.G];
            const int64_t n     = (int64_t) (args.M - first) * args.N;
            for (int64_t e = (int64_t) blockIdx.x * 128 + (threadIdx.x - 128); e < n; e += (int64_t) gridDim.x * 128)
                cbase[(first + e / args.N) * args.ldc + e % args.N] = from_f32<OutT>(0.0f);
        }
        uint32_t acc_it = 0;
        float acc[TN];
        while (ok && sched.get(t)) {
            const int gb   = args.kind == kKindGroupedRows ? t.g : 0;
            const int n    = t.n0 + quad * 32 + lane; // this lane's weight row = output column
            const int segs = kPerBlock ? t.num_kb : 1;
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[j] = 0.0f;
            for (int sidx = 0; sidx < segs; ++sidx, ++acc_it) {
                const uint32_t buf = acc_it % kAccBufs;
                const int slot     = acc_it % kScaleSlots;
                if constexpr (kPerBlock) {
                    if (!mbar_wait(smem_u32(&ctl->sc_full[slot]), (acc_it / kScaleSlots) & 1)) { ok = false; break; }
                }
                if (!mbar_wait(smem_u32(&ctl->tmem_full[buf]), (acc_it / kAccBufs) & 1)) { ok = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t) (quad * 32) << 16) + buf * TN;
                const float *sl      = &ctl->scale_ring[slot * kSlotFloats];
                const float sb       = kPerBlock ? sl[TN] : 1.0f;
#pragma unroll
                for (int c = 0; c < TN / 32; ++c) {
                    float v[32];
                    tc_ld32(taddr + 32 * c, v);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        float *d = &acc[32 * c + j];
                        if constexpr (kPerBlock) {
                            const float4 s4 = *reinterpret_cast<const float4 *>(sl + 32 * c + j);
                            d[0] = fmaf(v[j], s4.x * sb, d[0]);
                            d[1] = fmaf(v[j + 1], s4.y * sb, d[1]);
                            d[2] = fmaf(v[j + 2], s4.z * sb, d[2]);
                            d[3] = fmaf(v[j + 3], s4.w * sb, d[3]);
                        } else {
                            d[0] = v[j]; d[1] = v[j + 1]; d[2] = v[j + 2]; d[3] = v[j + 3];
                        }
                    }
                }
                tc_fence_before();
                __syncwarp(); // every lane has read the buffer and its scales
                if (lane == 0) {
                    mbar_arrive(smem_u32(&ctl->tmem_empty[buf]));
                    if constexpr (kPerBlock) mbar_arrive(smem_u32(&ctl->sc_empty[slot]));
                }
            }
            if (!ok) break;
            if (n < args.N) {
                float sw = 1.0f; // tensorwise: the whole factor; rowwise: this weight row's
                if constexpr (SCALE == kScaleTensor) sw = args.a_scale[0] * args.b_scale[0];
                if constexpr (SCALE == kScaleRow) sw = args.b_scale[(int64_t) gb * args.bs_g + (int64_t) n * args.bs_n];
                OutT *dst      = cbase + (int64_t) t.m0 * args.ldc + n;
                const int rows = min(TN, t.m_end - t.m0);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    if (j < rows) {
                        float v = acc[j];
                        if constexpr (SCALE == kScaleTensor) v *= sw;
                        if constexpr (SCALE == kScaleRow) v *= args.a_scale[(int64_t) (t.m0 + j) * args.as_m] * sw;
                        dst[(int64_t) j * args.ldc] = from_f32<OutT>(v);
                    }
                }
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicExch(&g_gemm_status, 3);
    }

    // ---- teardown ----
    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

template <int SCALE, typename OutT, int TN> int launch_skinny_tn(const GemmArgs &args, int grid, cudaStream_t st) {
    static bool configured[64] = {}; // per device; the attribute set is idempotent, a race only repeats it
    auto kfn = skinny_gemm_kernel<SCALE, OutT, TN>;
    int dev  = 0;
    PTB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        PTB_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) SkinnyGeo<TN>::kSmem));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    PTB_CUDA((launch_after(kfn, dim3((unsigned) grid), SkinnyGeo<TN>::kThreads, SkinnyGeo<TN>::kSmem, st, 1, args)));
    PTB_LAUNCH_CHECK("skinny_gemm_kernel");
    return 0;
}
template <int SCALE, typename OutT> int launch_skinny_out(const GemmArgs &args, int grid, cudaStream_t st) {
    switch (args.bm) {
    case 32: return launch_skinny_tn<SCALE, OutT, 32>(args, grid, st);
    case 64: return launch_skinny_tn<SCALE, OutT, 64>(args, grid, st);
    default: return launch_skinny_tn<SCALE, OutT, 128>(args, grid, st);
    }
}
template <int SCALE> int launch_skinny_scale(const GemmArgs &args, int out_dtype, int grid, cudaStream_t st) {
    switch (out_dtype) {
    case PTB_BF16: return launch_skinny_out<SCALE, __nv_bfloat16>(args, grid, st);
    case PTB_F16: return launch_skinny_out<SCALE, __half>(args, grid, st);
    case PTB_F32: return launch_skinny_out<SCALE, float>(args, grid, st);
    default: return fail(PTB_ERR_ARG, "GEMM output dtype %d is not supported", out_dtype);
    }
}

// Rows of `a` per tile for the swapped form, 0 where the 128 x 256 tile stays the better one.  Dense: all rows in one tile, so
// that the weight is read once; from 129 rows on the ordinary tile's 128-row side is full.
// Row groups: how the rows are spread is known on the device only, and a group of more than 32 rows reads its expert's
// weight once per 32.  So the line lies where a skewed load costs little: 32 experts x 4096 x 7168, tensorwise, ordinary
// against swapped, softmax loads of 8 rows a group 186 against 175 us, of 16 193 against 197; the same rows on two experts
// 53 against 59 and 57 against 98.  With block scales every further tile promotes its own partial products, and only
// calls that cannot give every SM an ordinary tile stay here (64 rows on two experts 46 against 38 us; softmax loads of 4,
// 12 and 24 rows a group 149, 187, 189 against 163, 210, 237).
int skinny_rows(int mode, int64_t rows, int64_t G, int64_t N, bool k_major, int grid) {
    if (!k_major || (mode != kScaleTensor && mode != kScaleRow && mode != kScaleBlock2D)) return 0;
    if (G == 0) return rows <= 32 ? 32 : rows <= 64 ? 64 : rows <= 128 ? 128 : 0;
    const bool few_tiles = rows * cdiv<int64_t>(N, kTileN) <= grid; // even if every row has an expert of its own
    return few_tiles || (mode != kScaleBlock2D && rows <= 8 * G) ? 32 : 0;
}

// `a` [M, K] and `w` [G or 1, N, K] (both K-major), as the entry points got them
int launch_skinny(GemmArgs &g, int mode, int tn, const void *a, int a_dtype, int64_t lda, const void *w, int w_dtype, int64_t ldw,
                  uint64_t groups, int out_dtype, int grid, cudaStream_t st) {
    set_tile(g, 1);
    g.bm = tn;
    g.bn = 128;
    int rc = make_map(&g.tm_a, a, (uint64_t) g.K, (uint64_t) g.M, 1, (uint64_t) lda, (uint64_t) lda * g.M, tn);
    if (rc) return rc;
    rc = make_map(&g.tm_b, w, (uint64_t) g.K, (uint64_t) g.N, groups, (uint64_t) ldw, (uint64_t) ldw * g.N, 128);
    if (rc) return rc;
    g.idesc   = make_idesc(w_dtype, a_dtype, 0, 0, tn); // the weight is the MMA's A operand
    g.tiles_n = (int) cdiv<int64_t>(g.N, 128);
    switch (mode) {
    case kScaleTensor: return launch_skinny_scale<kScaleTensor>(g, out_dtype, grid, st);
    case kScaleRow: return launch_skinny_scale<kScaleRow>(g, out_dtype, grid, st);
    default: return launch_skinny_scale<kScaleBlock2D>(g, out_dtype, grid, st);
    }
}

} // namespace
} // namespace ptb
