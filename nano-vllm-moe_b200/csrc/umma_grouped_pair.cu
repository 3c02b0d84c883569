// Grouped W8A8 GEMM of prefill-sized expert batches on CTA pairs (tcgen05 cta_group::2), channels as the MMA's M:
//
//   D[256 channels, T rows] = W_e[256 channels, K] . xq[rows of one chunk, K]^T        T = the chunk's rows, rounded up to 32
//
// for every chunk of at most 256 routed rows that share an expert e (chunk list of moe_align_kernel, rows already e4m3 and
// in sorted order) and every item of channels:
//   gate_up (kDown = false)  an item is gate tile t and up tile t of the expert (128 channels each).  CTA r of the pair takes
//             channels [64 r, 64 r + 64) of BOTH, so that a gate value and its up value meet in one CTA: warps of the gate
//             lanes and of the up lanes swap half of their values through shared memory and each finishes half the rows:
//             hq[sorted position][channel] = e4m3(h / h_scale), h = bf16(bf16(silu(g)) * u) from g, u rounded to bf16 (the
//             eager two-rounding SiluAndMul of the reference's experts).
//   down    (kDown = true)   an item is channel tiles 2 t and 2 t + 1, one per CTA; out[routed row][channel] =
//             bf16(acc * scale * routing weight).
//
// Tensor-bound.  Rows as the N dimension fit the work to the ragged row counts of the experts: 16384 rows over 60 experts are
// 2.1 chunks of 128 rows each as MMA M (384 of them multiplied for 273 on average) against 288 in steps of 32; and a pair
// moves 32 KB of operands into each SM per 256 x 256 x 128 block where one CTA needs 48 KB per 128 x 256 x 128.  Two accumulator
// stages of 256 columns let the epilogue of an item run under the next item's MMAs.
//
//   warp 0      TMA producer (both CTAs): 16 KB of weights and T/2 rows per K block
//   warp 1      MMA issuer (leader): four tcgen05.mma 256 x T x 32 per K block
//   warps 2..9  epilogue: warp (q, h) owns TMEM lanes [32 q, 32 q + 32) and half h of the rows
// All waits are bounded; the epilogue warps vote on each item, because they meet at named barriers.
#include "umma_common.cuh"

namespace fp8lin {

namespace {

constexpr int kStages = 6;
constexpr int kEpiWarps = 8;
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr int kKB = 128;
constexpr int kWBytes = 128 * kKB;                 // this CTA's 128 channel rows
constexpr int kXBytes = 128 * kKB;                 // up to 128 routed rows
constexpr int kStageBytes = kWBytes + kXBytes;
constexpr int kRingBytes = kStages * kStageBytes;
constexpr int kSwapBytes = 32 * 64;                // bf16 values of 32 rows x 32 channels, one buffer per warp pair
constexpr int kCodeBytes = 32 * 32;                // e4m3 of 32 rows x 32 channels
constexpr int kStagingBytes = 4 * (kSwapBytes + kCodeBytes);
constexpr int kSmemBytes = kRingBytes + kStagingBytes + 1024;
constexpr int kTmemCols = 512;
constexpr int kMaxT = 256;

__device__ __forceinline__ void bar_pair(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
// One chunk as every role sees it (values uniform over the warp).
struct Chunk {
    int expert, start, rows, tokens;
};
__device__ __forceinline__ Chunk load_chunk(const int4* chunks, int c) {
    const int4 v = chunks[c];
    Chunk r;
    r.expert = uniform(v.x);
    r.start = uniform(v.y);
    r.rows = uniform(v.z);
    r.tokens = (r.rows + 31) & ~31;
    return r;
}

// Boxes of the weights (64 rows for a half of gate_up, 128 for down; 16 for up rows inside tiles) and of 16, 32, .. 128 routed
// rows: a K block is two or three TMA instructions (with boxes of 64 and 16 rows, four to six, 2 % slower).
struct GroupedPairMaps {
    CUtensorMap w, w16, x[8];
};

template <bool kDown>
__global__ void __launch_bounds__(kThreads, 1)
grouped_pair_kernel(const __grid_constant__ GroupedPairMaps maps, GroupedArgs p) {
    constexpr int S = kStages;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[S];       // leader's: both CTAs' bytes
    __shared__ __align__(8) uint64_t bar_empty[S];
    __shared__ __align__(8) uint64_t bar_tfull[2];
    __shared__ __align__(8) uint64_t bar_tempty[2];     // leader's
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile int s_abort;
    __shared__ int s_routed[kMaxT];
    __shared__ float s_rw[kMaxT];

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) { mbar_init(smem_u32(&bar_full[i]), 1); mbar_init(smem_u32(&bar_empty[i]), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&bar_tfull[i]), 1); mbar_init(smem_u32(&bar_tempty[i]), 2 * kEpiWarps); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(smem_u32(&s_tmem_base), kTmemCols);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();            // the partner's barriers exist before anything is signalled on them
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    pdl_launch_dependents();
    pdl_wait();                    // the chunk list, the rows and the outputs all come from predecessors

    const int n_chunks = uniform(p.meta[0]);
    const int n_items = p.n_tiles;                    // channel items per chunk (set by the launcher)
    const int total = n_chunks * n_items;             // work w = chunk * n_items + item
    const int first = (int)(blockIdx.x >> 1), step = (int)(gridDim.x >> 1);
    const int KB = p.kblocks;

    if (warp == 0) {
        // ================= TMA producer (both CTAs) =================
        const uint32_t el = elect_one();
        int st = 0;
        uint32_t phase = 1;                           // parity that a free slot shows on its first use
        bool ok = true;
        for (int w = first; w < total && ok; w += step) {
            const Chunk ch = load_chunk(p.chunks, w / n_items);
            const int t = w % n_items;
            const int half = ch.tokens >> 1;          // rows of this CTA: a multiple of 16
            const int row0 = ch.start + (int)rank * half;
            const CUtensorMap* x_map = &maps.x[(half >> 4) - 1];
            const uint32_t bytes = (uint32_t)(kWBytes + half * kKB);
            // packed weight rows of K block 0: gate_up 64 rows each of gate tile t and up tile t; down its own tile (the last
            // item of an odd number of tiles has none for CTA 1: it multiplies tile 2 t again and stores nothing)
            const int tile_a = kDown ? min(2 * t + (int)rank, p.w_tiles - 1) : t;
            const int wrow_a = (ch.expert * p.w_tiles + tile_a) * KB * 128 + (kDown ? 0 : (int)rank * 64);
            // up channels start at row N of the expert's weight, perhaps inside a tile: then four boxes of 16 rows, which a
            // tile boundary (N is a multiple of 16) never cuts
            const int up_row = p.N + t * 128 + (int)rank * 64;
            const bool up_whole = (p.N & 63) == 0;
            int wrow_b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                wrow_b[i] = (ch.expert * p.w_tiles + ((up_row + 16 * i) >> 7)) * KB * 128 + ((up_row + 16 * i) & 127);
            for (int kb = 0; kb < KB; ++kb) {
                ok = __all_sync(0xffffffffu, !s_abort && mbar_wait(smem_u32(&bar_empty[st]), phase, p.status, kDevTimeoutEmpty));
                if (!ok) { s_abort = 1; break; }
                const uint32_t full_local = smem_u32(&bar_full[st]);
                mbar_expect_tx(leader ? el : 0u, full_local, 2 * bytes);
                const uint32_t full = map_to_cta(full_local, 0);
                const uint32_t sa = smem_base + st * kStageBytes;
                tma_load_2d_pair(el, sa, &maps.w, 0, wrow_a + kb * 128, full);             // 64 rows of gate, or all 128 of down
                if (!kDown) {
                    if (up_whole) tma_load_2d_pair(el, sa + kWBytes / 2, &maps.w, 0, wrow_b[0] + kb * 128, full);
                    else {
#pragma unroll
                        for (int i = 0; i < 4; ++i) tma_load_2d_pair(el, sa + kWBytes / 2 + i * 2048, &maps.w16, 0, wrow_b[i] + kb * 128, full);
                    }
                }
                const uint32_t sx = sa + kWBytes;
                tma_load_2d_pair(el, sx, x_map, kb * kKB, row0, full);
                if (++st == S) { st = 0; phase ^= 1; }
            }
        }
        if (!ok) {
            const long long t0 = clock64();           // let copies that are still in flight land
            while (clock64() - t0 < 2000000) {}
        }
    } else if (warp == 1) {
        // ================= MMA issuer (leader CTA only) =================
        if (leader) {
            const uint32_t el = elect_one();
            constexpr uint16_t both = 3;
            int st = 0, tl = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int w = first; w < total && ok; w += step, ++tl) {
                const Chunk ch = load_chunk(p.chunks, w / n_items);
                const uint32_t idesc = make_idesc_mn(256, ch.tokens, 0, 0);
                const int as = tl & 1;
                const uint32_t aph = (tl >> 1) & 1;
                ok = __all_sync(0xffffffffu, !s_abort && mbar_wait(smem_u32(&bar_tempty[as]), aph ^ 1, p.status, kDevTimeoutTmemEmpty));
                if (!ok) { s_abort = 1; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * kMaxT;
                for (int kb = 0; kb < KB; ++kb) {
                    ok = __all_sync(0xffffffffu, !s_abort && mbar_wait(smem_u32(&bar_full[st]), phase, p.status, kDevTimeoutFull));
                    if (!ok) { s_abort = 1; break; }
                    tc_fence_after();
                    const uint32_t sa = smem_base + st * kStageBytes;
                    const uint64_t da = make_smem_desc(sa);
                    const uint64_t db = make_smem_desc(sa + kWBytes);
#pragma unroll
                    for (int k = 0; k < kKB / 32; ++k) umma_f8_pair(el, d_tmem, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit_both(el, smem_u32(&bar_empty[st]), both);
                    if (++st == S) { st = 0; phase ^= 1; }
                }
                if (ok) umma_commit_both(el, smem_u32(&bar_tfull[as]), both);
            }
        }
    } else {
        // ================= epilogue (warps 2..9 of both CTAs) =================
        const int q = warp & 3;                       // TMEM lane quarter
        const int h = (warp - 2) >> 2;                // half of the chunk's rows
        const int et = threadIdx.x - 64;              // 0..255 among the epilogue threads
        const float in_scale = fmaxf(__ldg(p.input_scale), 1e-12f);
        const ExactDiv div_h(kDown ? 1.f : fmaxf(__ldg(p.h_scale), 1e-12f));
        const bool up = q >= 2;                       // gate_up: lanes of quarters 2, 3 are up channels
        const int pair = (q & 1) + 2 * h;             // the warps of quarters q and q ^ 2 share 32 channels and a buffer
        const uint32_t swap_buf = smem_base + kRingBytes + pair * (kSwapBytes + kCodeBytes);
        const uint32_t code_buf = swap_buf + kSwapBytes;
        // output channel of this lane (gate_up: of the pair of values) and its multiplier
        auto channel_of = [&](int t) { return kDown ? (2 * t + (int)rank) * 128 + q * 32 + lane : t * 128 + (int)rank * 64 + (q & 1) * 32 + lane; };
        auto scale_of = [&](int e, int n) -> float {
            if (n >= p.N) return 0.f;
            return in_scale * __ldg(p.w_scale + (kDown ? (size_t)e * p.N + n : (size_t)e * 2 * p.N + (up ? p.N : 0) + n));
        };
        int next_routed = 0;
        float next_rw = 0.f, next_scale = 0.f;
        auto prefetch = [&](int w) {                  // row `et` of the chunk, this lane's multiplier
            const Chunk c = load_chunk(p.chunks, w / n_items);
            next_scale = scale_of(c.expert, channel_of(w % n_items));
            if (kDown && et < c.rows) {
                next_routed = __ldg(p.sorted_rows + c.start + et);
                next_rw = __ldg(p.topk_w + next_routed);
            }
        };
        if (first < total) prefetch(first);
        int tl = 0;
        for (int w = first; w < total; w += step, ++tl) {
            const Chunk ch = load_chunk(p.chunks, w / n_items);
            const int n = channel_of(w % n_items);
            const float scale = next_scale;
            const int as = tl & 1;
            const uint32_t aph = (tl >> 1) & 1;
            if (kDown) {
                if (tl > 0) asm volatile("bar.sync 5, 256;" ::: "memory");        // the previous item's rows have been used
                s_routed[et] = next_routed;
                s_rw[et] = next_rw;
            }
            if (w + step < total) prefetch(w + step);
            const bool arrived = mbar_wait(smem_u32(&bar_tfull[as]), aph, p.status, kDevTimeoutTmemFull);
            uint32_t any_failed;                      // publishes the rows and takes the vote: the eight warps leave together
            asm volatile(
                "{\n .reg .pred pin, pout;\n setp.ne.b32 pin, %1, 0;\n"
                " barrier.cta.red.or.pred pout, 5, 256, pin;\n selp.u32 %0, 1, 0, pout;\n}"
                : "=r"(any_failed) : "r"(arrived ? 0u : 1u) : "memory");
            if (any_failed) { s_abort = 1; break; }
            tc_fence_after();
            const int half = ch.tokens >> 1;
            const int m0 = h * half;                  // first row (of the chunk) of this warp
            const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + as * kMaxT + m0;
            const int used = min(half, ch.rows - m0); // rows of this warp that exist (the same for both warps of a pair)
            auto release = [&]() {                    // the accumulator is in registers: the next item but one may have it
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(&bar_tempty[as]), 0));
            };
            if (used <= 0) release();
            for (int c = 0; c < used; c += 32) {
                const int n_cols = min(32, half - c); // 32 or 16
                uint32_t v[32];
                __syncwarp();
                tmem_ld32_nowait(t_addr + c, v);
                tmem_ld_wait();
                if (c + 32 >= used) release();
                if constexpr (kDown) {
                    // two lanes swap halves: an even lane stores two channels of the even rows, an odd lane of the odd rows
                    const bool odd = lane & 1;
                    const bool in = (n & ~1) < p.N;
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        if (j == 16 && n_cols == 16) break;
                        const int m = m0 + c + j + (odd ? 1 : 0);
                        const float rw0 = s_rw[m0 + c + j], rw1 = s_rw[m0 + c + j + 1];
                        const float a0 = __uint_as_float(v[j]) * scale * rw0, a1 = __uint_as_float(v[j + 1]) * scale * rw1;
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 1);
                        const uint32_t o = odd ? pack_bf16x2(other, a1) : pack_bf16x2(a0, other);
                        if (in && m < ch.rows) *reinterpret_cast<uint32_t*>(p.out + (size_t)s_routed[m] * p.ld_out + (n & ~1)) = o;
                    }
                } else {
                    // Values as the bf16 gate_up row.  The gate warp finishes columns [0, 16) of the 32, the up warp [16, 32): each
                    // hands the other half over.  No branches inside (a last piece of 16 columns computes 16 more that are not
                    // stored), so that the eight chains of exp and divisions overlap.
                    uint32_t own[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t lo = pack_bf16x2(__uint_as_float(v[2 * j]) * scale, __uint_as_float(v[2 * j + 1]) * scale);
                        const uint32_t hi = pack_bf16x2(__uint_as_float(v[16 + 2 * j]) * scale, __uint_as_float(v[16 + 2 * j + 1]) * scale);
                        own[j] = up ? hi : lo;
                        const uint32_t give = up ? lo : hi;
                        // (column pairs as words: [pair][lane], the gate's half in front)
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(swap_buf + (up ? 0 : 1024) + j * 128 + lane * 4), "r"(give) : "memory");
                    }
                    bar_pair(1 + pair);
                    uint32_t other[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(other[j]) : "r"(swap_buf + (up ? 1024 : 0) + j * 128 + lane * 4) : "memory");
                    const uint32_t code_at = code_buf + (up ? 16 * 32 : 0) + lane;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t g = up ? other[j] : own[j], u = up ? own[j] : other[j];
                        const float g0 = bf16_lo(g), g1 = bf16_hi(g);
                        const uint32_t sv = pack_bf16x2(silu_f32(g0), silu_f32(g1));              // bf16(silu(g))
                        const uint32_t hv = pack_bf16x2(bf16_lo(sv) * bf16_lo(u), bf16_hi(sv) * bf16_hi(u));          // bf16(. * u)
                        const uint32_t code = cvt_e4m3x2(div_h(bf16_lo(hv)), div_h(bf16_hi(hv)));
                        asm volatile("st.shared.u8 [%0], %1;" ::"r"(code_at + 2 * j * 32), "r"(code & 0xffu) : "memory");
                        asm volatile("st.shared.u8 [%0], %1;" ::"r"(code_at + (2 * j + 1) * 32), "r"(code >> 8) : "memory");
                    }
                    bar_pair(1 + pair);
                    // 32 bytes per row: thread i of the 64 stores half a row
                    const int i = (up ? 32 : 0) + lane;
                    const int m = m0 + c + (i >> 1);
                    if ((i >> 1) < n_cols && m < ch.rows && (n - lane) + (i & 1) * 16 < p.N) {      // (N is a multiple of 16)
                        const float4 o = ld_shared_f4(code_buf + (i >> 1) * 32 + (i & 1) * 16);
                        *reinterpret_cast<float4*>(p.hq + (size_t)(ch.start + m) * p.N + (n - lane) + (i & 1) * 16) = o;
                    }
                }
            }
        }
    }

    // nobody leaves while its partner may still signal its barriers or the leader's MMAs may still read its shared memory and
    // write its tensor memory
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

template <bool kDown>
cudaError_t launch_kernel(const GroupedArgs& a, const GroupedPairMaps& maps, cudaStream_t stream, const char** why) {
    auto kern = grouped_pair_kernel<kDown>;
    static SmemOptIn opted;
    cudaError_t e = ensure_dynamic_smem((const void*)kern, kSmemBytes, opted);
    if (e != cudaSuccess) return e;
    const int pairs = max_active_clusters((const void*)kern, kThreads, kSmemBytes, 2);
    if (pairs < 1) {
        if (why) *why = "no CTA pair fits on this device";
        return cudaErrorInvalidConfiguration;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = pdl_attribute(attr);
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 2;
    attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = na + 1;
    return counted(cudaLaunchKernelEx(&cfg, kern, maps, a));
}

}  // namespace

cudaError_t launch_grouped_pair_w8a8(GroupedArgs a, const void* w_packed, int num_experts, const void* xq_sorted, int64_t xq_rows,
                                     cudaStream_t stream, const char** why) {
    const bool gate_up = a.hq != nullptr;                          // a.N = I gate channels; the expert's weight holds 2 I channels
    const int tiles = (int)pack_ntiles(a.N);
    a.w_tiles = (int)pack_ntiles(gate_up ? 2 * (int64_t)a.N : a.N);
    a.kblocks = (int)pack_kblocks(a.K);
    a.n_tiles = gate_up ? tiles : (tiles + 1) / 2;
    if (a.N % 16 != 0 || (!gate_up && a.ld_out % 2 != 0)) {
        if (why) *why = "the output width must be a multiple of 16";
        return cudaErrorInvalidValue;
    }
    GroupedPairMaps maps;
    const uint64_t w_rows = (uint64_t)num_experts * a.w_tiles * a.kblocks * 128;
    bool ok = encode_u8_2d(&maps.w, w_packed, w_rows, 128, gate_up ? 64 : 128) && encode_u8_2d(&maps.w16, w_packed, w_rows, 128, 16);
    for (int i = 0; i < 8 && ok; ++i) ok = encode_u8_2d(&maps.x[i], xq_sorted, (uint64_t)xq_rows, (uint64_t)a.K, 16 * (i + 1));
    if (!ok) {
        if (why) *why = "cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    return gate_up ? launch_kernel<false>(a, maps, stream, why) : launch_kernel<true>(a, maps, stream, why);
}

}  // namespace fp8lin
