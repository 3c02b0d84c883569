// W8A8 linear on CTA pairs (tcgen05 cta_group::2), operands swapped, for batches between decode and prefill and for row
// counts that do not fill 256-row tiles:
//
//   y^T[N, M] = W_e4m3[N, K] . xq_e4m3[M, K]^T          fp32 accumulation in TMEM
//
// A pair of CTAs computes 256 output channels x T tokens.  CTA r of the pair owns channels [128 r, 128 r + 128) of the tile
// (the weight tile is its half of the MMA's "A" operand) and stages T/2 of the rows of xq as its half of "B".  The rows are
// the MMA's N, so a tile takes any multiple of 32 of them up to 256, and the last tile of the batch may be smaller than the
// others: 1031 rows are 4 x 256 + 32 of them instead of 5 x 256.
//
//   warp 0        TMA producer: 16 KB of weights and T/2 x 128 bytes of xq per slot; the weights of the first ring pass go
//                 out before the wait for the kernel that writes xq
//   warp 1        MMA issuer (leader CTA): four tcgen05.mma.cta_group::2.kind::f8f6f4 (256 x T x 32) per K block
//   warps 2..9    epilogue: lane = channel, y[m][n] = bf16(acc * in_scale * w_scale[n] + bias[n]), turned to rows in shared memory
//
// kMlp (gate_up of the fused MLP, gate and up channels in alternating tiles of 128): a CTA stages 64 gate channels and the
// 64 up channels of the same indices, and the epilogue writes e4m3 h = bf16(silu(g) * u) / h_scale; the warps of the gate
// lanes and of the up lanes swap half of their values and finish half of the rows each.
//
// The caller says into how many slices the K blocks of a sum are cut: a slice is accumulated by itself and the slices are
// added in order, which makes the result the same bits as that of the kernel that would otherwise take the call (the decode
// kernels up to 64 rows, the one-CTA GEMM above).  Two ways:
//   one pair works through all slices, each into its own T columns of tensor memory, and the epilogue adds them
//   kSplit (few tiles, long K): the 2 s CTAs of a cluster take one slice each of the same tile
//   and park their sums in shared memory; slice r's CTA adds up band r of its pair rank's channels
//
// What bounds it: up to T = 64 the way of 16 KB of weights per CTA and K block into shared memory (0.09 us when few SMs load,
// 0.16 when all do), above that the tensor core (512 cycles per K block at T = 256), for large calls its power.  Per call on
// codes, in a loop over weights from memory, us: decode kernel, one-CTA GEMM or 256-row pairs, whichever would be chosen / here
// with the lanes storing the results / here: 3584 -> 3584 64 rows 7.07 / 7.25 / 6.92, 256 rows 9.8 / 8.5 / 8.2; 3584 -> 4608 1031 rows 19.9 / 16.8
// / 16.1; 3584 -> 37888 1031 rows 122 / 110 / 107 (power: 5 % from run to run); 18944 -> 3584 700 rows 54 / 41.3 / 40.9, 1031 rows
// 60 / 54.6 / 53.7.  All waits are bounded.
#include "umma_common.cuh"

namespace fp8lin {

namespace {

constexpr int kEpiWarps = 8;
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr int kTile = 128;                     // channels per CTA
constexpr int kKB = 128;                       // K elements per block
constexpr int kWBytes = kTile * kKB;
constexpr int kMaxSlots = 12;
constexpr int kMaxT = 256;                     // columns of an accumulator stage
constexpr int kTmemCols = 512;
template <bool kStored> constexpr int kRingBytes = (kStored ? 200 : 210) * 1024;       // 16 KB + 64 T bytes per slot; kStored: beside boxes
constexpr int kBoxBytes = 32 * 128;            // results of 32 tokens x 64 channels on their way out, one box per two epilogue warps
constexpr int kSwapBytes = 32 * 64;            // kMlp: bf16 values of 32 rows x 32 channels, one buffer per warp pair
constexpr int kCodeBytes = 32 * 32;            // ... and their e4m3 results
template <bool kSplit, bool kMlp>
constexpr int kSmemBytes = kRingBytes<!kSplit && !kMlp> + 4 * (kMlp ? kSwapBytes + kCodeBytes : kSplit ? 0 : kBoxBytes) + 1024;
static_assert(kTile * 256 * 4 <= kRingBytes<false>, "the parked sums must fit in the ring");

struct PairSched8 {
    int n_tiles;              // 256-channel tiles
    int m_tiles;              // token tiles
    int tokens, last_tokens;  // T of all token tiles but the last, and of the last
    int slices;               // K slices of a sum
    int splits;               // kSplit: = slices (cluster of 2 * slices CTAs); else 1: persistent over all tiles
    int kblocks, kblocks_per_slice;
};

// weights (boxes of 128 rows, kMlp 64), xq (boxes of half a full and half a last token tile) and y (16 tokens x 64 channels)
struct PairMaps8 {
    CUtensorMap w, x, x_last, y;
};

struct Item {
    int nt;                   // channel tile
    int m0, half;             // first token, half of its tokens
    bool last;
};
// Token tiles of a channel tile follow each other, so that its weights come from L2 after the first; every other channel tile
// walks them backwards, or with an even number of token tiles the same pairs would always get the last, smaller ones.
__device__ __forceinline__ Item decode_item(const PairSched8& s, int item) {
    Item r;
    r.nt = item / s.m_tiles;
    int mi = item - r.nt * s.m_tiles;
    if (r.nt & 1) mi = s.m_tiles - 1 - mi;
    r.last = mi == s.m_tiles - 1;
    r.m0 = mi * s.tokens;
    r.half = (r.last ? s.last_tokens : s.tokens) >> 1;
    return r;
}

// A sum times in_scale, then times the channel's scale: in two roundings up to 64 rows, as the decode kernels do it, in one
// product of the scales above, as the 256-row kernels do.  The bf16 results of a row count are the same bits whichever kernel
// takes it.  Returns the factor of the channel's scale; `pre` multiplies the sum.
__device__ __forceinline__ float channel_factor(const UmmaArgs& p, float& pre) {
    const float in_scale = fmaxf(ld_dep(p.input_scale), 1e-12f);
    pre = p.M <= 64 ? in_scale : 1.f;
    return p.M <= 64 ? 1.f : in_scale;
}

template <bool kSplit, bool kMlp>
__global__ void __launch_bounds__(kThreads, 1)
w8a8_pair_kernel(const __grid_constant__ PairMaps8 maps, UmmaArgs p, PairSched8 sched) {
    static_assert(!(kSplit && kMlp), "the activation epilogue takes whole sums");
    constexpr int kRing = kRingBytes<!kSplit && !kMlp>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kMaxSlots];      // leader's: both CTAs' weights and rows landed
    __shared__ __align__(8) uint64_t bar_empty[kMaxSlots];     // the MMAs that read the slot are done (both CTAs')
    __shared__ __align__(8) uint64_t bar_tfull[2];
    __shared__ __align__(8) uint64_t bar_tempty[2];            // leader's
    __shared__ __align__(8) uint64_t bar_done;                 // tensor memory of both CTAs has been read for the last time
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile int s_abort;

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    const uint32_t crank = cluster_ctarank();
    const uint32_t rank = crank & 1;                   // inside the pair
    const bool leader = rank == 0;
    const uint32_t leader_cta = crank & ~1u;
    const int slice_rank = kSplit ? (int)(crank >> 1) : 0;
    const int items = sched.n_tiles * sched.m_tiles;
    const int first_item = kSplit ? (int)(blockIdx.x / (2 * sched.splits)) : (int)(blockIdx.x >> 1);
    const int item_step = kSplit ? items : (int)(gridDim.x >> 1);
    const int kb0 = slice_rank * sched.kblocks_per_slice;
    const int kb1 = kSplit ? min(sched.kblocks, kb0 + sched.kblocks_per_slice) : sched.kblocks;
    // accumulators: `slices` times T columns per tile, two tiles where they fit
    const int n_acc = kSplit ? 1 : sched.slices;
    const int acc_cols = n_acc * sched.tokens;
    const int acc_stages = 2 * acc_cols <= kTmemCols ? 2 : 1;
    const uint32_t slot_bytes = kWBytes + (uint32_t)sched.tokens * 64u;
    const int n_slots = min(kMaxSlots, (int)(kRing / slot_bytes));
    // split-K: band r of this CTA's 128 channels is finished by slice r's CTA of the same pair rank
    const int band = kSplit ? (kTile + sched.splits - 1) / sched.splits : kTile;
    const int band_rows = kSplit ? max(0, min(kTile, (slice_rank + 1) * band) - slice_rank * band) : 0;
    const Item it0 = decode_item(sched, first_item);
    const int m_valid = kSplit ? min(2 * it0.half, p.M - it0.m0) : 0;
    // split-K: this CTA's raw sums lie over the (then idle) ring as [group of four tokens][channel], 16 bytes each, so that 32
    // lanes (channels) touch 512 contiguous bytes.  The CTA that finishes a band fetches its channels from all slices.
    // Sent to it by st.async instead (which suits the few rows of the decode kernels), 128 channels x T sums took longer: 256 rows on
    // 18944 -> 3584 22.2 us against 20.9.
    constexpr uint32_t group_bytes = kParkedGroupBytes;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kMaxSlots; ++i) { mbar_init(smem_u32(&bar_full[i]), 1); mbar_init(smem_u32(&bar_empty[i]), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&bar_tfull[i]), 1); mbar_init(smem_u32(&bar_tempty[i]), 2 * kEpiWarps); }
        mbar_init(smem_u32(&bar_done), 2 * kEpiWarps);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    const uint32_t el = elect_one();
    auto load_weights = [&](const Item& it, int kb, int slot) {
        const uint32_t full_local = smem_u32(&bar_full[slot]);
        mbar_expect_tx(leader ? el : 0u, full_local, 2u * (kWBytes + (uint32_t)it.half * kKB));
        const uint32_t full = map_to_cta(full_local, leader_cta);
        const uint32_t ws = smem_base + slot * slot_bytes;
        if (kMlp) {
            const int row = (2 * it.nt * sched.kblocks + kb) * kTile + (int)rank * 64;
            tma_load_2d_pair(el, ws, &maps.w, 0, row, full);
            tma_load_2d_pair(el, ws + kWBytes / 2, &maps.w, 0, row + sched.kblocks * kTile, full);
        } else {
            tma_load_2d_pair(el, ws, &maps.w, 0, ((2 * it.nt + (int)rank) * sched.kblocks + kb) * kTile, full);
        }
    };
    pair_enter();
    const int pre = min(kb1 - kb0, n_slots);               // K blocks of the first ring pass
    if (warp == 0)
        for (int i = 0; i < pre; ++i) load_weights(it0, kb0 + i, i);
    const uint32_t tmem_base = pair_tmem_begin(warp, &s_tmem_base, kTmemCols);
    pdl_launch_dependents();

    if (warp == 0) {
        // ================= TMA producer (both CTAs) =================
        auto load_rows = [&](const Item& it, int kb, int slot) {
            const uint32_t full = map_to_cta(smem_u32(&bar_full[slot]), leader_cta);
            tma_load_2d_pair(el, smem_base + slot * slot_bytes + kWBytes, it.last ? &maps.x_last : &maps.x, kb * kKB, it.m0 + (int)rank * it.half, full);
        };
        pdl_wait();
        for (int i = 0; i < pre; ++i) load_rows(it0, kb0 + i, i);
        int slot = pre == n_slots ? 0 : pre;
        uint32_t phase = pre == n_slots ? 0 : 1;           // parity that a free slot shows (1 on its first use)
        bool ok = true;
        for (int item = first_item; item < items && ok; item += item_step) {
            const Item it = decode_item(sched, item);
            for (int kb = item == first_item ? kb0 + pre : kb0; kb < kb1; ++kb) {
                ok = !s_abort && warp_wait(smem_u32(&bar_empty[slot]), phase, p.status, kDevTimeoutEmpty);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; s_abort = 1; break; }
                load_weights(it, kb, slot);
                load_rows(it, kb, slot);
                if (++slot == n_slots) { slot = 0; phase ^= 1; }
            }
        }
        if (!ok) {
            const long long t0 = clock64();                // let copies that are still in flight land
            while (clock64() - t0 < 2000000) {}
        }
    } else if (warp == 1) {
        // ================= MMA issuer (leader CTA only) =================
        if (leader) {
            const uint16_t both = (uint16_t)(3u << crank);                      // this CTA and its partner
            int tl = 0, slot = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int item = first_item; item < items && ok; item += item_step, ++tl) {
                const Item it = decode_item(sched, item);
                const uint32_t idesc = make_idesc_mn(2 * kTile, 2 * it.half, 0, 0);          // e4m3 x e4m3
                const int as = acc_stages == 2 ? (tl & 1) : 0;
                const uint32_t aph = acc_stages == 2 ? ((tl >> 1) & 1) : (tl & 1);
                ok = __all_sync(0xffffffffu, !s_abort && mbar_wait<true>(smem_u32(&bar_tempty[as]), aph ^ 1, p.status, kDevTimeoutTmemEmpty));
                if (!ok) { s_abort = 1; break; }
                tc_fence_after();
                uint32_t d_tmem = tmem_base + as * acc_cols;
                int left = sched.kblocks_per_slice;           // K blocks until the next slice's accumulator
                bool fresh = true;
                for (int kb = kb0; kb < kb1; ++kb) {
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[slot]), phase, p.status, kDevTimeoutFull));
                    if (!ok) { s_abort = 1; break; }
                    tc_fence_after();
                    const uint64_t da = make_smem_desc(smem_base + slot * slot_bytes);
                    const uint64_t db = make_smem_desc(smem_base + slot * slot_bytes + kWBytes);
#pragma unroll
                    for (int k = 0; k < kKB / 32; ++k)
                        umma_f8_pair(el, d_tmem, da + 2 * k, db + 2 * k, idesc, (!fresh || k > 0) ? 1u : 0u);
                    umma_commit_both(el, smem_u32(&bar_empty[slot]), both);
                    fresh = false;
                    if (--left == 0) { left = sched.kblocks_per_slice; d_tmem += sched.tokens; fresh = true; }
                    if (++slot == n_slots) { slot = 0; phase ^= 1; }
                }
                if (ok) umma_commit_both(el, smem_u32(&bar_tfull[as]), both);
            }
        }
        if (!kSplit) pair_tmem_release(smem_u32(&bar_done), tmem_base, kTmemCols, p.status);
    } else {
        // ================= epilogue (warps 2..9 of both CTAs) =================
        pdl_wait();                                        // the output may still be in use by the predecessor
        const int q = warp & 3;                            // TMEM lane quarter
        const int h = (warp - 2) >> 2;                     // which half of the tile's tokens
        float pre;
        const float in_scale = channel_factor(p, pre);
        const ExactDiv div_h(kMlp ? fmaxf(ld_dep(p.h_scale), 1e-12f) : 1.f);
        const bool odd = lane & 1;
        const bool up = kMlp && q >= 2;
        const int pair = (q & 1) + 2 * h;                  // kMlp: the warps of quarters q and q ^ 2 share 32 channels
        const uint32_t swap_buf = smem_base + kRing + pair * (kSwapBytes + kCodeBytes);
        const uint32_t code_buf = swap_buf + kSwapBytes;
        int tl = 0;
        for (int item = first_item; item < items; item += item_step, ++tl) {
            const Item it = decode_item(sched, item);
            const int as = acc_stages == 2 ? (tl & 1) : 0;
            // this lane's channel as the weights are laid out
            const int n = kMlp ? it.nt * 256 + (up ? 128 : 0) + (int)rank * 64 + (q & 1) * 32 + lane : (2 * it.nt + (int)rank) * kTile + q * 32 + lane;
            float ws = 0.f, bs = 0.f;
            if (!kSplit && n < p.N) {
                ws = in_scale * ld_dep(p.w_scale + n);
                if (p.bias) bs = ld_dep(p.bias + n);
            }
            bool arrived = mbar_wait(smem_u32(&bar_tfull[as]), acc_stages == 2 ? ((tl >> 1) & 1) : (tl & 1), p.status, kDevTimeoutTmemFull);
            if (!kSplit) arrived = !named_sync_any(5, 256, !arrived);      // warps that meet at barriers below leave together
            if (!arrived) { s_abort = 1; break; }
            tc_fence_after();
            const int m0 = it.m0 + h * it.half;
            const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16) + as * acc_cols + h * it.half;
            auto read32 = [&](int c, uint32_t* v) {        // columns [c, c + 32) or, at the end of the tile, [c, c + 16)
                __syncwarp();
                tmem_ld16_nowait(t_lane + c, v);
                if (c + 16 < it.half) tmem_ld16_nowait(t_lane + c + 16, v + 16);
                tmem_ld_wait();
                for (int sl = 1; sl < n_acc; ++sl) {       // the other slices, in order
                    uint32_t u[32];
                    tmem_ld16_nowait(t_lane + sl * sched.tokens + c, u);
                    if (c + 16 < it.half) tmem_ld16_nowait(t_lane + sl * sched.tokens + c + 16, u + 16);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(u[j]));
                }
                if (!kSplit && c + 32 >= it.half) {        // all in registers: the next tile but one may have the accumulator
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(&bar_tempty[as]), leader_cta));
                }
            };
            if constexpr (kMlp) {
                const int hc = it.nt * 128 + (int)rank * 64 + (q & 1) * 32;           // first of the 32 output channels
                const int ld = p.N >> 1;
                for (int c = 0; c < it.half; c += 32) {
                    uint32_t v[32];
                    read32(c, v);
                    const int n_cols = min(32, it.half - c);
                    uint32_t lo[8], hi[8];                 // the bf16 values that a separate gate_up linear stores
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        lo[j] = pack_bf16x2(fmaf(__uint_as_float(v[2 * j]) * pre, ws, bs), fmaf(__uint_as_float(v[2 * j + 1]) * pre, ws, bs));
                        hi[j] = pack_bf16x2(fmaf(__uint_as_float(v[16 + 2 * j]) * pre, ws, bs), fmaf(__uint_as_float(v[16 + 2 * j + 1]) * pre, ws, bs));
                    }
                    gate_up_swap<32, false>(lo, hi, up, swap_buf, code_buf, 1 + pair, lane, div_h);
                    const int i = (up ? 32 : 0) + lane;                               // 32 bytes per row: a thread stores half a row
                    const int m = m0 + c + (i >> 1);
                    if ((i >> 1) < n_cols && m < p.M)
                        *reinterpret_cast<float4*>(p.hq + (size_t)m * ld + hc + (i & 1) * 16) = ld_shared_f4(code_buf + (i >> 1) * 32 + (i & 1) * 16);
                }
            } else if constexpr (!kSplit) {
                // Two warps (64 channels) fill a box of 32 tokens, which leaves by TMA in whole 128-byte lines, clipped at M and N
                // (stored by the lanes, 64 bytes of a row at a time, the tile of T = 224 took 6600 SM cycles behind the last MMA, 2500 of
                // them for the stores).  Two lanes swap halves, so that a lane writes two channels of a token: even lanes token j, odd lanes j + 4, whose
                // swizzled places lie in the other banks.
                const uint32_t box = smem_base + kRing + ((q >> 1) + 2 * h) * kBoxBytes;
                const bool issuer = (q & 1) == 0 && lane == 0;
                const int n_box = (2 * it.nt + (int)rank) * kTile + (q >> 1) * 64;
                const uint32_t at = box + (odd ? 512u : 0u) + (uint32_t)(lane & 6) * 2u, chunk = (uint32_t)((q & 1) * 4 + (lane >> 3)), sel = odd ? 0x3276u : 0x5410u;
                for (int c = 0; c < it.half; c += 32) {
                    uint32_t v[32];
                    read32(c, v);
                    uint32_t o[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int k = 8 * (j >> 2) + (j & 3);
                        o[j] = pack_bf16x2(fmaf(__uint_as_float(v[k]) * pre, ws, bs), fmaf(__uint_as_float(v[k + 4]) * pre, ws, bs));
                        o[j] = __byte_perm(o[j], __shfl_xor_sync(0xffffffffu, o[j], 1), sel);
                    }
                    if (issuer) tma_store_wait_read();         // the previous store has read the box
                    named_sync(1 + (q >> 1) + 2 * h, 64);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {             // row 8 (j / 4) + j % 4, odd lanes four further on
                        const uint32_t r = (uint32_t)(j & 3) + (odd ? 4u : 0u);
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + (uint32_t)(8 * (j >> 2) + (j & 3)) * 128u + ((chunk ^ r) << 4)), "r"(o[j]) : "memory");
                    }
                    fence_async_smem();
                    named_sync(1 + (q >> 1) + 2 * h, 64);
                    if (issuer && n_box < p.N) {
                        if (m0 + c < p.M) tma_store_2d(&maps.y, box, n_box, m0 + c);
                        if (c + 16 < it.half && m0 + c + 16 < p.M) tma_store_2d(&maps.y, box + kBoxBytes / 2, n_box, m0 + c + 16);
                    }
                }
            } else {
                // the pair's MMAs are done, so this CTA's ring is free
                const uint32_t dst = smem_base + (uint32_t)(h * it.half >> 2) * group_bytes + (uint32_t)(q * 32 + lane) * 16u;
                for (int c = 0; c < it.half; c += 32) {
                    uint32_t v[32];
                    read32(c, v);
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        if (j == 16 && c + 16 >= it.half) break;
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (uint32_t)((c + j) >> 2) * group_bytes), "r"(v[j]), "r"(v[j + 1]),
                                     "r"(v[j + 2]), "r"(v[j + 3]) : "memory");
                    }
                }
            }
        }
        pair_tmem_done(smem_u32(&bar_done), leader_cta, lane);
        if (!kSplit && !kMlp && lane == 0) tma_store_wait_all();
    }

    if constexpr (kSplit) {
        // ---- this CTA finishes its band: slices added in rank order, scaled, stored ----
        __syncwarp();
        pdl_wait();
        cluster_sync_all();                                // every CTA's sums are parked
        if (warp == 1) pair_tmem_release(smem_u32(&bar_done), tmem_base, kTmemCols, p.status);
        if (!s_abort) {
            float pre;
            const float in_scale = channel_factor(p, pre);
            finish_parked_band(p, smem_base, sched.splits, (int)rank, slice_rank * band, band_rows, m_valid, (2 * it0.nt + (int)rank) * kTile,
                               it0.m0, pre, in_scale, kThreads);
        }
    }

    pair_leave();
}

template <bool kSplit, bool kMlp>
cudaError_t launch_kernel(const W8a8PairPlan& pl, const UmmaArgs& a, const PairMaps8& maps, cudaStream_t stream) {
    auto kern = w8a8_pair_kernel<kSplit, kMlp>;
    static SmemOptIn opted;
    cudaError_t e = ensure_dynamic_smem((const void*)kern, kSmemBytes<kSplit, kMlp>, opted);
    if (e != cudaSuccess) return e;
    PairSched8 s;
    s.n_tiles = pl.n_tiles; s.m_tiles = pl.m_tiles; s.tokens = pl.tokens; s.last_tokens = pl.last_tokens; s.splits = pl.splits; s.slices = pl.slices;
    s.kblocks = (a.K + kKB - 1) / kKB; s.kblocks_per_slice = (s.kblocks + s.slices - 1) / s.slices;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)pl.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes<kSplit, kMlp>;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = pdl_attribute(attr);
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = (unsigned)(2 * pl.splits);
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return counted(cudaLaunchKernelEx(&cfg, kern, maps, a, s));
}

}  // namespace

// Tokens per tile, and whether a cluster takes the slices: the cheapest by a model of the kernel in microseconds, fitted to
// back-to-back calls with every T and 1 to 4 slices over twelve layer shapes (1280 -> 1536 .. 2048 -> 11008 .. 18944 -> 3584, 3584
// -> 37888) at 16 to 4096 rows while the lanes stored the results; with the results by TMA the choice of T is 0.3 % slower than the best of
// the sweep on average where the kernel is routed to (eleven shapes, 17 to 3000 rows), 0.7 % over all of them.  A K block takes the longer
// of the way of the operands into shared memory (0.09 + 0.0003 T: 16 KB of weights whatever T is; more when every SM loads)
// and the tensor core's (0.03 + 0.0013 T); all blocks together at least what the power limit allows.  A call starts later the
// more SMs it needs at once (the kernel before it is still on them), and clusters add the hand-over of the sums and their
// start: they only pay for long K, and are only taken when all fit at once.
W8a8PairPlan plan_w8a8_pair(int64_t M, int64_t K, int64_t N, bool mlp, int slices, int force_tokens, int force_splits) {
    W8a8PairPlan best{};
    best.cost = 1e30;
    const int kblocks = (int)((K + kKB - 1) / kKB);
    const int n_tiles = (int)((N + 255) / 256);
    if (slices < 1 || slices > 8 || slices > kblocks) return best;
    const int kps = (kblocks + slices - 1) / slices;
    if ((kblocks + kps - 1) / kps != slices) return best;                     // would leave an empty slice
    for (int pass = 0; pass < 2; ++pass) {
        const int splits = pass == 0 ? 1 : slices;
        if (pass == 1 && (slices == 1 || slices > 4 || mlp)) break;
        if (force_splits > 0 && splits != force_splits) continue;
        const void* kern = splits > 1 ? (const void*)w8a8_pair_kernel<true, false>
                         : mlp ? (const void*)w8a8_pair_kernel<false, true> : (const void*)w8a8_pair_kernel<false, false>;
        const int slots = max_active_clusters(kern, kThreads, splits > 1 ? kSmemBytes<true, false> : mlp ? kSmemBytes<false, true> : kSmemBytes<false, false>, 2 * splits);
        if (slots < 1) continue;
        const int blocks = splits > 1 ? kps : kblocks;                        // K blocks of a pair
        for (int tokens = 32; tokens <= kMaxT; tokens += 32) {
            if (force_tokens > 0 && tokens != force_tokens) continue;
            if (force_tokens <= 0 && tokens >= M + 32) break;
            if (splits == 1 && slices * tokens > kTmemCols) break;
            const int m_tiles = (int)((M + tokens - 1) / tokens);
            const int last = (int)((M - (int64_t)(m_tiles - 1) * tokens + 31) / 32) * 32;
            const long items = (long)n_tiles * m_tiles;
            if (force_splits <= 0 && splits > 1 && items > slots) continue;
            const long rounds = (items + slots - 1) / slots;
            const double active = (double)(items < slots ? items : slots) * splits, pairs = sm_count() / 2;
            const double load = active / pairs;
            const double hbm = 32768.0 * active / m_tiles / 10.7e6;           // (the other token tiles find the weights in L2)
            auto block = [&](int t) {
                const double in = (0.0907 + 0.00029 * t) * (1.0 + 0.755 * load), mma = 0.0323 + 0.00126 * t * (1.0 + 0.175 * load);
                const double own = in > mma ? in : mma;
                return own > hbm ? own : hbm;
            };
            const double t_last = block(last), t_full = m_tiles > 1 ? block(tokens) : t_last;
            const double mean = ((m_tiles - 1) * t_full + t_last) / m_tiles;
            const double drain = 0.0122 * tokens + (splits > 1 ? 0.0 : 0.2 * (slices - 1));
            double chain = blocks * (rounds == 1 ? t_full : rounds * mean);
            if (splits == 1 && 2 * slices * tokens > kTmemCols) chain += (rounds - 1) * drain;      // one accumulator stage
            const double power = (double)n_tiles * kblocks / pairs * ((m_tiles - 1) * (0.148 + 0.0009 * tokens) + 0.148 + 0.0009 * last);
            if (power > chain) chain = power;
            static const double cluster_start[5] = {0, 0, 0.92, 0.51, 0.67};
            const double tail = splits > 1 ? 0.96 + cluster_start[splits] + 0.030 * tokens * (1.0 - 1.0 / splits) : drain;
            const double cost = chain + 1.66 + 1.53 * load + tail;
            if (cost < best.cost) {
                best.cost = cost;
                best.n_tiles = n_tiles; best.m_tiles = m_tiles; best.tokens = tokens; best.last_tokens = last;
                best.slices = slices; best.splits = splits;
                best.grid = splits > 1 ? (int)(items * 2 * splits) : 2 * (int)(items < slots ? items : slots);
            }
        }
    }
    return best;
}

cudaError_t launch_w8a8_pair(const W8a8PairPlan& pl, const UmmaArgs& a, cudaStream_t stream, const char** why) {
    const bool mlp = a.hq != nullptr;
    PairMaps8 maps;
    bool ok = pl.tokens >= 32 && encode_u8_2d(&maps.w, a.w, (uint64_t)(pack_ntiles(a.N) * pack_kblocks(a.K) * 128), 128, mlp ? kTile / 2 : kTile) &&
              encode_u8_2d(&maps.x_last, a.xq, (uint64_t)a.M, (uint64_t)a.K, (uint32_t)pl.last_tokens / 2);
    maps.x = maps.x_last;                                  // (a map costs the host 0.1 us: only what the kernel reads)
    if (ok && pl.m_tiles > 1 && pl.tokens != pl.last_tokens) ok = encode_u8_2d(&maps.x, a.xq, (uint64_t)a.M, (uint64_t)a.K, (uint32_t)pl.tokens / 2);
    maps.y = maps.x_last;
    if (ok && !mlp && pl.splits == 1) ok = encode_out_2d(&maps.y, a.y, (uint64_t)a.M, (uint64_t)a.N, (uint64_t)a.ldy * 2, 64, 16);
    if (!ok) {
        if (why) *why = "no plan, or cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    if (mlp) return launch_kernel<false, true>(pl, a, maps, stream);
    return pl.splits > 1 ? launch_kernel<true, false>(pl, a, maps, stream) : launch_kernel<false, false>(pl, a, maps, stream);
}

}  // namespace fp8lin
