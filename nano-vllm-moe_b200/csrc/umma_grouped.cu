// Grouped W8A8 GEMM for the MoE expert FFN on tcgen05 (operands swapped, as in umma_swap.cu):
// for every chunk of up to MP routed rows that share an expert e and every 128-channel tile t
//
//     D[128 channels, MP rows] = W_e[tile t, K] . xq[rows, K]^T
//
// The expert's weight tile is the 128-row MMA "A" operand (TMA, packed layout, one 16 KiB box
// per K block); the routed rows are the MMA "N" dimension.  Work items (chunk, tile) come from
// the chunk list that the grouping (moe_kernels.cu) leaves in device memory, so no host synchronisation is needed;
// the grid is persistent (one CTA per SM) and every CTA strides over the items.
//
// Source of the rows (template flag kGather):
//   true   decode-sized batches of the gate_up projection: the rows are gathered from the bf16
//          token matrix through the sorted row index and quantised on the fly (static scale,
//          exact division) by converter warps straight into the swizzled MMA "B" tile.
//   false  the rows are already e4m3 and contiguous in sorted order (down projection always;
//          gate_up after moe_place_kernel for prefill-sized batches): one TMA box.
// Epilogue (run-time flag `scatter`):
//   0      gu[sorted position][channel] = bf16(acc * in_scale * w_scale[e][channel])
//   1      out[routed row][channel] = bf16(acc * in_scale * w_scale[e][channel] * topk_w[routed row])
//
// kFused (gate_up): the 128 rows of a weight tile are 64 gate channels and the 64 up channels of the same indices, so that a
// work item holds both halves of 64 outputs and the epilogue writes what the down projection reads instead of bf16 gate_up
// rows: hq[sorted position][channel] = e4m3(h / h_scale) with h = bf16(bf16(silu(g)) * u) from g, u rounded to bf16 -- the
// values and roundings of the separate activation pass (the eager two-rounding SiluAndMul of the reference's experts).  The
// warps of the gate lanes and of the up lanes swap half of their values through shared memory and finish half of the rows
// each.  Any intermediate size that is a multiple of 16.  Saves the bf16 tensor and a launch of the decode step's chain
// (64 tokens, 4 of 60 experts, hidden 2048, intermediate 1408, back to back: 101 -> 99 us per block).
//
// Weight-bandwidth-bound for small batches (each expert's weights are read once per chunk),
// tensor-bound for prefill-sized batches.  All mbarrier waits are bounded.
#include "umma_common.cuh"

namespace fp8lin {

constexpr int kGrpConvWarps = 8;
constexpr int kGrpThreads = (2 + kGrpConvWarps + 4) * 32;
constexpr int kGrpTile = 128;
constexpr int kGrpKB = 128;

template <int MP, bool kFused = false>
struct GroupedCfg {
    static constexpr int kWBytes = kGrpTile * kGrpKB;
    static constexpr int kXqBytes = MP * kGrpKB;
    static constexpr int kStageBytes = kWBytes + kXqBytes;
    static constexpr int kStagesRaw = (218 * 1024) / kStageBytes;
    static constexpr int kStages = kStagesRaw > 10 ? 10 : kStagesRaw;
    static constexpr int kSmemBytes = kStages * kStageBytes + 1024;
    static constexpr int kAccCols = MP;                            // TMEM columns of one accumulator stage
    static constexpr int kTmemCols = 2 * kAccCols < 32 ? 32 : 2 * kAccCols;
    static constexpr int kTeam = MP <= 16 ? 1 : (MP <= 32 ? 2 : 4);
    static constexpr int kPiece = MP < 32 ? MP : 32;            // accumulator columns per TMEM read
    static_assert(kStageBytes % 1024 == 0, "stage alignment");
};

// Boxes of the weights: 128 rows (plain), or 64 (fused; 16 where the up rows lie inside tiles); rows of xq: MP.
struct GroupedMaps {
    CUtensorMap w, w16, xq;
};

template <int MP, bool kGather, bool kFused = false>
__global__ void __launch_bounds__(kGrpThreads, 1)
grouped_w8a8_kernel(const __grid_constant__ GroupedMaps maps, GroupedArgs p) {
    using Cfg = GroupedCfg<MP, kFused>;
    constexpr int S = Cfg::kStages;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[S];
    __shared__ __align__(8) uint64_t bar_xq[S];
    __shared__ __align__(8) uint64_t bar_empty[S];
    __shared__ __align__(8) uint64_t bar_tfull[2];
    __shared__ __align__(8) uint64_t bar_tempty[2];
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile int s_abort;
    constexpr int kSwapWords = kFused ? 2 * Cfg::kPiece * 16 : 1;              // bf16 pairs of kPiece rows x 32 channels, per warp pair
    __shared__ __align__(16) uint32_t s_swap[kSwapWords];
    __shared__ __align__(16) unsigned char s_code[kFused ? 2 * Cfg::kPiece * 32 : 16];

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = warp_index();
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(smem_u32(&bar_full[i]), 1);
            mbar_init(smem_u32(&bar_xq[i]), Cfg::kTeam);
            mbar_init(smem_u32(&bar_empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&bar_tfull[i]), 1); mbar_init(smem_u32(&bar_tempty[i]), 4); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(&s_tmem_base), Cfg::kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    pdl_launch_dependents();
    pdl_wait();                                   // the chunk list, the rows and the outputs all come from predecessors

    const int n_chunks = uniform(p.meta[0]);
    const int total = n_chunks * p.n_tiles;       // item w = chunk * n_tiles + tile
    const int KB = p.kblocks;

    if (warp == 0) {
        // ================= TMA producer =================
        {
            const uint32_t el = elect_one();
            if (el) {
                asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.w) : "memory");
                if (!kGather) asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.xq) : "memory");
            }
            uint32_t it = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
                const int4 chunk = p.chunks[w / p.n_tiles];
                const int2 ch = make_int2(uniform(chunk.x), uniform(chunk.y));
                const int t = w % p.n_tiles;
                // packed row of K block 0: tile t, or (fused) 64 gate channels and their up channels
                const int wrow0 = kFused ? ((ch.x * p.w_tiles + (t >> 1)) * KB) * kGrpTile + (t & 1) * 64 : ((ch.x * p.w_tiles + t) * KB) * kGrpTile;
                const int up_row = p.N + t * 64;
                const bool up_whole = (p.N & 63) == 0;
                int wrow_up[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    wrow_up[i] = ((ch.x * p.w_tiles + ((up_row + 16 * i) >> 7)) * KB) * kGrpTile + ((up_row + 16 * i) & 127);
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int st = it % S;
                    const uint32_t ph = (it / S) & 1;
                    ok = __all_sync(0xffffffffu, !s_abort && mbar_wait(smem_u32(&bar_empty[st]), ph ^ 1, p.status, kDevTimeoutEmpty));
                    if (!ok) { s_abort = 1; break; }
                    const uint32_t full = smem_u32(&bar_full[st]);
                    const uint32_t sa = smem_base + st * Cfg::kStageBytes;
                    mbar_expect_tx(el, full, kGather ? Cfg::kWBytes : Cfg::kWBytes + Cfg::kXqBytes);
                    tma_load_2d(el, sa, &maps.w, 0, wrow0 + kb * kGrpTile, full);
                    if (kFused) {
                        if (up_whole) tma_load_2d(el, sa + Cfg::kWBytes / 2, &maps.w, 0, wrow_up[0] + kb * kGrpTile, full);
                        else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) tma_load_2d(el, sa + Cfg::kWBytes / 2 + i * 2048, &maps.w16, 0, wrow_up[i] + kb * kGrpTile, full);
                        }
                    }
                    if (!kGather) tma_load_2d(el, sa + Cfg::kWBytes, &maps.xq, kb * kGrpKB, ch.y, full);
                }
            }
            if (!ok) {
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) {}
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        {
            const uint32_t el = elect_one();
            constexpr uint32_t idesc = make_idesc_mn(kGrpTile, MP, 0, 0);
            uint32_t it = 0;
            int tl = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < total && ok; w += gridDim.x, ++tl) {
                const int as = tl & 1;
                const uint32_t aph = (tl >> 1) & 1;
                ok = __all_sync(0xffffffffu, !s_abort && mbar_wait(smem_u32(&bar_tempty[as]), aph ^ 1, p.status, kDevTimeoutTmemEmpty));
                if (!ok) { s_abort = 1; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * Cfg::kAccCols;
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int st = it % S;
                    const uint32_t ph = (it / S) & 1;
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[st]), ph, p.status, kDevTimeoutFull) &&
                                                     (!kGather || mbar_wait(smem_u32(&bar_xq[st]), ph, p.status, kDevTimeoutFull)));
                    if (!ok) { s_abort = 1; break; }
                    tc_fence_after();
                    const uint32_t sa = smem_base + st * Cfg::kStageBytes;
                    const uint64_t da = make_smem_desc(sa);
                    const uint64_t db = make_smem_desc(sa + Cfg::kWBytes);
#pragma unroll
                    for (int k = 0; k < kGrpKB / 32; ++k) umma_f8(el, d_tmem, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit(el, smem_u32(&bar_empty[st]));
                }
                if (ok) umma_commit(el, smem_u32(&bar_tfull[as]));
            }
        }
    } else if (warp < 2 + kGrpConvWarps) {
        // ================= row gather + quantise (gate_up flavour only) =================
        if (kGather) {
            constexpr int kTeams = kGrpConvWarps / Cfg::kTeam;
            const int team = (warp - 2) / Cfg::kTeam;       // a ring slot always belongs to the same team
            const int member = (warp - 2) % Cfg::kTeam;
            const ExactDiv div_scale(fmaxf(ld_dep(p.input_scale), 1e-12f));
            uint32_t it = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
                const int4 ch = p.chunks[w / p.n_tiles];
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int st = it % S;
                    if (st % kTeams != team) continue;
                    const uint32_t ph = (it / S) & 1;
                    // the slot's previous MMAs must be done before its "B" tile is overwritten
                    if (s_abort || !mbar_wait(smem_u32(&bar_empty[st]), ph ^ 1, p.status, kDevTimeoutEmpty)) {
                        s_abort = 1; ok = false; break;
                    }
                    const uint32_t xq = smem_base + st * Cfg::kStageBytes + Cfg::kWBytes;
                    for (int i = member * 32 + lane; i < MP * 8; i += 32 * Cfg::kTeam) {
                        const int r = i >> 3, c = i & 7;
                        const int k = kb * kGrpKB + c * 16;
                        uint2 qa = make_uint2(0u, 0u), qb = make_uint2(0u, 0u);
                        if (r < ch.z && k < p.K) {
                            const int src_row = ld_dep(p.sorted_rows + ch.y + r) / p.x_div;
                            const uint4* src = reinterpret_cast<const uint4*>(p.x + (size_t)src_row * p.ldx + k);
                            qa = quant8_e4m3(ld_dep(src), div_scale);
                            qb = quant8_e4m3(ld_dep(src + 1), div_scale);
                        }
                        const uint32_t dst = xq + r * 128 + (((uint32_t)c ^ (uint32_t)(r & 7)) << 4);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(qa.x), "r"(qa.y), "r"(qb.x),
                                     "r"(qb.y) : "memory");
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&bar_xq[st]));
                }
            }
        }
    } else {
        // ================= epilogue (warps 10..13) =================
        const int q = warp & 3;
        const float in_scale = fmaxf(ld_dep(p.input_scale), 1e-12f);
        int tl = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < total && ok; w += gridDim.x, ++tl) {
            const int4 ch = p.chunks[w / p.n_tiles];
            const int t = w % p.n_tiles;
            const int as = tl & 1;
            const uint32_t aph = (tl >> 1) & 1;
            // output channel of this lane and its multiplier (fused: lanes of quarters 2, 3 hold the up values of the channels
            // of quarters 0, 1)
            const bool up = kFused && q >= 2;
            const int n = kFused ? t * 64 + (q & 1) * 32 + lane : t * kGrpTile + q * 32 + lane;
            const float ws = n < p.N ? in_scale * ld_dep(p.w_scale + (kFused ? (size_t)ch.x * 2 * p.N + (up ? p.N : 0) : (size_t)ch.x * p.N) + n) : 0.f;
            // routed-row index and routing weight of the chunk's rows, one row per lane and piece;
            // the inner loop gets them by shuffle instead of two dependent global loads per row
            int my_routed[(MP + 31) / 32];
            float my_w[(MP + 31) / 32];
#pragma unroll
            for (int i = 0; i < (MP + 31) / 32; ++i) {
                const int r = i * 32 + lane;
                my_routed[i] = 0; my_w[i] = 0.f;
                if (p.scatter && r < ch.z) {
                    my_routed[i] = ld_dep(p.sorted_rows + ch.y + r);
                    my_w[i] = ld_dep(p.topk_w + my_routed[i]);
                }
            }
            bool arrived = mbar_wait(smem_u32(&bar_tfull[as]), aph, p.status, kDevTimeoutTmemFull);
            if (kFused) arrived = !named_sync_any(3, 128, !arrived);              // warps that meet at barriers below leave together
            if (!arrived) { s_abort = 1; ok = false; break; }
            tc_fence_after();
            const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + as * Cfg::kAccCols;
            if constexpr (kFused) {
                constexpr int kP = Cfg::kPiece, kH = kP / 4;      // rows per step; column pairs each warp of a pair finishes
                const ExactDiv div_h(fmaxf(ld_dep(p.h_scale), 1e-12f));
                const uint32_t swap_buf = smem_u32(s_swap) + (uint32_t)(q & 1) * (kP * 64);
                const uint32_t code_buf = smem_u32(s_code) + (uint32_t)(q & 1) * (kP * 32);
#pragma unroll 1
                for (int c0 = 0; c0 < MP; c0 += kP) {
                    if (c0 >= ch.z) break;                        // the same for both warps of a pair
                    uint32_t v[kP];
                    __syncwarp();
                    if (kP == 32) tmem_ld32_nowait(t_addr + c0, v);
                    else tmem_ld16_nowait(t_addr + c0, v);
                    tmem_ld_wait();
                    uint32_t lo[kH], hi[kH];                      // as the bf16 gate_up row
#pragma unroll
                    for (int j = 0; j < kH; ++j) {
                        lo[j] = pack_bf16x2(__uint_as_float(v[2 * j]) * ws, __uint_as_float(v[2 * j + 1]) * ws);
                        hi[j] = pack_bf16x2(__uint_as_float(v[kP / 2 + 2 * j]) * ws, __uint_as_float(v[kP / 2 + 2 * j + 1]) * ws);
                    }
                    gate_up_swap<kP, true>(lo, hi, up, swap_buf, code_buf, 1 + (q & 1), lane, div_h);
                    // 32 bytes per row: thread i of the 64 stores half a row (N is a multiple of 16)
                    const int i = (up ? 32 : 0) + lane, r = i >> 1, nh = (n - lane) + (i & 1) * 16;
                    if (r < kP && c0 + r < ch.z && nh < p.N)
                        *reinterpret_cast<float4*>(p.hq + (size_t)(ch.y + c0 + r) * p.N + nh) = ld_shared_f4(code_buf + r * 32 + (i & 1) * 16);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[as]));
                continue;
            }
#pragma unroll 1
            for (int c0 = 0; c0 < MP; c0 += Cfg::kPiece) {
                if (c0 >= ch.z) break;                                           // uniform: no rows left in this chunk
                uint32_t v[Cfg::kPiece];
                __syncwarp();
                if (Cfg::kPiece == 32) tmem_ld32_nowait(t_addr + c0, v);
                else tmem_ld16_nowait(t_addr + c0, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < Cfg::kPiece; ++j) {
                    const int r = c0 + j;                                       // uniform across the warp
                    const int routed = __shfl_sync(0xffffffffu, my_routed[(c0 + j) / 32], (c0 + j) & 31);
                    const float rw = __shfl_sync(0xffffffffu, my_w[(c0 + j) / 32], (c0 + j) & 31);
                    if (r < ch.z && n < p.N) {
                        const float acc = __uint_as_float(v[j]) * ws;
                        if (!p.scatter) p.out[(size_t)(ch.y + r) * p.ld_out + n] = __float2bfloat16_rn(acc);
                        else p.out[(size_t)routed * p.ld_out + n] = __float2bfloat16_rn(acc * rw);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[as]));
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

// ---- host side -------------------------------------------------------------------
template <int MP, bool kGather, bool kFused = false>
static cudaError_t launch_grouped(const GroupedArgs& a, const GroupedMaps& maps, cudaStream_t stream) {
    using Cfg = GroupedCfg<MP, kFused>;
    auto kern = grouped_w8a8_kernel<MP, kGather, kFused>;
    static SmemOptIn opted;
    {
        cudaError_t e = ensure_dynamic_smem((const void*)kern, Cfg::kSmemBytes, opted);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count());
    cfg.blockDim = dim3(kGrpThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.numAttrs = pdl_attribute(attr);
    cfg.attrs = attr;
    return counted(cudaLaunchKernelEx(&cfg, kern, maps, a));
}

int grouped_chunk_rows(int64_t rows, int num_experts) {
    const int64_t avg = num_experts > 0 ? (rows + num_experts - 1) / num_experts : rows;
    return avg <= 16 ? 16 : (avg <= 32 ? 32 : (avg <= 64 ? 64 : 128));
}

cudaError_t launch_grouped_w8a8(bool gather, int mp, GroupedArgs a, const void* w_packed, int num_experts,
                                const void* xq_sorted, int64_t xq_rows, cudaStream_t stream, const char** why) {
    GroupedMaps maps;
    const bool fused = a.hq != nullptr;           // a.N = I gate channels; the expert's weight holds 2 I channels
    a.n_tiles = fused ? (a.N + 63) / 64 : (int)pack_ntiles(a.N);
    a.w_tiles = (int)pack_ntiles(fused ? 2 * (int64_t)a.N : a.N);
    a.kblocks = (int)pack_kblocks(a.K);
    const uint64_t w_rows = (uint64_t)num_experts * a.w_tiles * a.kblocks * 128;
    if (!encode_u8_2d(&maps.w, w_packed, w_rows, 128, fused ? 64 : kGrpTile) || !encode_u8_2d(&maps.w16, w_packed, w_rows, 128, 16)) {
        if (why) *why = "cuTensorMapEncodeTiled failed for the expert weights";
        return cudaErrorInvalidValue;
    }
    maps.xq = maps.w;
    if (!gather && !encode_u8_2d(&maps.xq, xq_sorted, (uint64_t)xq_rows, (uint64_t)a.K, (uint32_t)mp)) {
        if (why) *why = "cuTensorMapEncodeTiled failed for the quantised rows";
        return cudaErrorInvalidValue;
    }
#define FP8LIN_GROUPED_CASE(MP_)                                                                                               \
    if (mp == MP_) {                                                                                                           \
        if (gather) return fused ? launch_grouped<MP_, true, true>(a, maps, stream) : launch_grouped<MP_, true>(a, maps, stream); \
        return fused ? launch_grouped<MP_, false, true>(a, maps, stream) : launch_grouped<MP_, false>(a, maps, stream);          \
    }
    FP8LIN_GROUPED_CASE(16)
    FP8LIN_GROUPED_CASE(32)
    FP8LIN_GROUPED_CASE(64)
    FP8LIN_GROUPED_CASE(128)
#undef FP8LIN_GROUPED_CASE
    if (why) *why = "unsupported chunk size";
    return cudaErrorInvalidValue;
}

}  // namespace fp8lin
