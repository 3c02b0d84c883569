// W8A16 linear on CTA pairs (tcgen05 cta_group::2), operands swapped, weights widened on the way to the tensor cores:
//
//   y^T[N, M] = bf16(W_e4m3[N, K]) . x[M, K]^T          fp32 accumulation in TMEM
//
// A pair of CTAs computes 256 output channels x T tokens (T = 32..256, a multiple of 32).  CTA r of the pair owns channels
// [128 r, 128 r + 128): its e4m3 weight tile arrives by TMA, converter warps widen it in registers to bf16 (exact) and put
// it into TENSOR MEMORY, where the MMA takes its "A" operand from; the bf16 activations are the caller's own rows, T/2 of
// them per CTA by TMA (128-byte swizzle) as the "B" operand.  So the weights cross HBM and L2 once as bytes, nothing is
// written back widened, and no pass over x is needed (the earlier route for more than 64 rows re-read the weights for
// every 64 rows on mma.sync, and from 256 rows wrote f16 copies of weights and activations to scratch first).
//
// What bounds it: per 128-element K block a CTA widens 16 KB of weights (about 400 SM cycles on the ALU and FMA pipes,
// eight warps) and the tensor core works 4 T cycles, so up to T = 160 the weight stream (690 cycles per 16 KB at 6.5 TB/s
// over 148 SMs) or the widening is the limit and above it the tensor core.  Against one CTA with the same T the pair
// halves the activation bytes each SM stages and feeds to its tensor core, which shared memory could not carry (a 128 x
// 256 tile would move 160 KB per 1024 cycles).
//
//   warp 0        activation producer: TMA of this CTA's half of the tokens, 128 K elements per slot
//   warp 18       weight producer: TMA of this CTA's 16 KB tiles, as many slots as fit
//   warps 2..9    two converter teams of four warps (one warp per 32-lane quarter of TMEM) taking turns: a lane widens one
//                 weight row, 2 x 64 codes -> 2 x 32 words -> tcgen05.st
//   warp 1        MMA issuer (leader CTA): eight tcgen05.mma.cta_group::2.kind::f16 (256 x T x 16) per K block
//   warps 10..17  epilogue: lane = channel, y[m][n] = bf16(acc * w_scale[n] + bias[n]); two lanes swap halves so that a lane
//                 stores two channels of one token
//
// Few tiles: the K blocks are cut into up to four slices, the 2 s CTAs of a cluster take one slice each of the same tile and
// park their sums in shared memory, and the CTA of slice r adds up band r of its pair rank's channels, slices in rank order (so
// results do not depend on timing).  All waits are bounded.
#include "umma_common.cuh"

namespace fp8lin {

namespace {

constexpr int kMaxA = 6;                       // widened weight tiles in TMEM (tmem_plan)
constexpr int kMaxW = 12, kMaxX = 12;          // slots of the weight and of the activation ring (ring_slots)
constexpr int kConvWarps = 8;
constexpr int kEpiWarps = 8;
constexpr int kThreads = (3 + kConvWarps + kEpiWarps) * 32;
constexpr int kTile = 128;                     // channels per CTA
constexpr int kKB = 128;                       // K elements per block
constexpr int kWBytes = kTile * kKB;           // 16 KB of codes
constexpr int kRingBytes = 216 * 1024;         // activation ring (128 T bytes per slot and CTA) and weight ring (16 KB per slot)
constexpr int kSmemBytes = kRingBytes + 1024;
constexpr int kACols = 64;                     // 128 bf16 of a row = 64 columns
constexpr int kTmemCols = 512;
static_assert(kTile * 256 * 4 <= kRingBytes, "the parked sums must fit in the ring");

// Ring depths for T tokens per tile.  A slot is occupied from its TMA until its MMAs (activations) or its widening (weights)
// are done, an L2 / HBM round trip of 1 to 1.5 us under load plus the chain through converters and tensor core, so with
// four activation slots a 16 KB weight block took 0.72 us whatever T was.  The activations get about half of the room, up to
// 12 slots, the weights the rest (five slots at T = 256).
__host__ __device__ inline void ring_slots(int tokens, int& nx, int& nw) {
    const int xb = 128 * tokens;
    nx = kRingBytes * 5 / 9 / xb;
    if (nx > kMaxX) nx = kMaxX;
    if (nx < 4) nx = 4;
    nw = (kRingBytes - nx * xb) / kWBytes;
    if (nw > kMaxW) nw = kMaxW;
}

// Tensor memory: accumulators from column 0 (two stages of T columns where that leaves room for four widened weight tiles,
// else one), widened tiles of 64 columns behind them.
__host__ __device__ inline void tmem_plan(int tokens, int& acc_stages, int& na) {
    acc_stages = tokens <= 128 ? 2 : 1;
    na = (kTmemCols - acc_stages * tokens) / kACols;
    if (na > kMaxA) na = kMaxA;
}

struct PairSched16 {
    int n_tiles;          // 256-channel tiles
    int m_tiles;          // token tiles
    int tokens;           // T
    int splits;           // K slices (cluster of 2 * splits CTAs); 1 = persistent over all tiles
    int kblocks, kblocks_per_split;
};

// 32 consecutive TMEM columns of this lane <- 32 registers; no wait
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr),
          "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Two e4m3 codes of a word -> bf16x2, exact.  The magnitude bits go to bits 4..10 of a bf16 and the sign stays in bit 15; that bf16 is
// the code's value times 2^-120 (e4m3 subnormals become bf16 subnormals), so one multiplication by 2^120 finishes it.  The byte
// permutation replicates the sign bit, so that a shift (as a product: the ALU is the busier pipe) and a mask are all there is between.
// With the sign put in by a second product instead, 64 rows on 3584 -> 37888 32.1 -> 30.3 us, 100 rows 37.5 -> 35.4.  (Four teams
// of converters instead of two: the same; the sums of the NaN test as products too: slower.)  The NaN codes 0x7f / 0xff come out as
// +-480; the caller tests for them.
template <uint32_t kSelector>                      // 0x9180: codes 0 and 1 of the word, 0xb3a2: 2 and 3 (bit 3 of a digit: the byte's sign)
__device__ __forceinline__ uint32_t e4m3_pair_to_bf16(uint32_t codes) {
    uint32_t q, r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(q) : "r"(codes), "n"(kSelector));
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"((q * 16u) & 0x87f087f0u), "r"(0x7b807b80u));
    return r;
}

__device__ __forceinline__ uint4 ld_shared_u4(uint32_t addr) {
    uint4 w;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(addr));
    return w;
}

// Half a weight row (64 codes: chunks 4 half .. 4 half + 3 of the swizzled 128-byte row) -> 32 words of bf16x2.
__device__ __forceinline__ void widen_half_row(uint32_t row_addr, uint32_t swizzle, int half, uint32_t* v) {
    uint32_t bad = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint4 w = ld_shared_u4(row_addr + ((((uint32_t)(4 * half + c)) ^ swizzle) << 4));
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[8 * c + 2 * j] = e4m3_pair_to_bf16<0x9180>(u[j]);
            v[8 * c + 2 * j + 1] = e4m3_pair_to_bf16<0xb3a2>(u[j]);
            bad |= (u[j] & 0x7f7f7f7fu) + 0x01010101u;               // bit 7 of a byte: its code was a NaN
        }
    }
    if (bad & 0x80808080u) {                                          // never in a checkpoint that quantised finite weights
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint4 w = ld_shared_u4(row_addr + ((((uint32_t)(4 * half + c)) ^ swizzle) << 4));
            const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (((u[j] >> (8 * b)) & 0x7fu) == 0x7fu) v[8 * c + 2 * j + (b >> 1)] |= 0x7fffu << (16 * (b & 1));
            }
        }
    }
}

template <bool kSplit>
__global__ void __launch_bounds__(kThreads, 1)
w8a16_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, UmmaArgs p, PairSched16 sched) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_wfull[kMaxW];    // this CTA's weight tile landed
    __shared__ __align__(8) uint64_t bar_wempty[kMaxW];   // ... and has been widened (four warps of the owning team)
    __shared__ __align__(8) uint64_t bar_xfull[kMaxX]; // leader's: both CTAs' activation blocks landed
    __shared__ __align__(8) uint64_t bar_xempty[kMaxX];// ... and the MMAs that read them are done (both CTAs')
    __shared__ __align__(8) uint64_t bar_conv[kMaxA];     // leader's: widened weights of both CTAs are in TMEM
    __shared__ __align__(8) uint64_t bar_empty[kMaxA];    // the MMAs that read the widened weights are done (both CTAs')
    __shared__ __align__(8) uint64_t bar_tfull[2];
    __shared__ __align__(8) uint64_t bar_tempty[2];    // leader's
    __shared__ __align__(8) uint64_t bar_done;         // tensor memory of both CTAs has been used for the last time
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
    const int kb0 = slice_rank * sched.kblocks_per_split;
    const int kb1 = kSplit ? min(sched.kblocks, kb0 + sched.kblocks_per_split) : sched.kblocks;
    const int T = sched.tokens;
    const int half = T >> 1;                           // tokens per CTA (a multiple of 16)
    int acc_stages, n_a;
    tmem_plan(T, acc_stages, n_a);
    const uint32_t a_col0 = (uint32_t)(acc_stages * T);
    const uint32_t x_bytes = (uint32_t)half * 256u;    // one activation block of this CTA: two 64-element halves
    const uint32_t xhalf_bytes = x_bytes >> 1;
    int nx, nw;
    ring_slots(T, nx, nw);
    const uint32_t wring = smem_base + nx * x_bytes;
    // split-K: band r of this CTA's 128 channels is finished by slice r's CTA of the same pair rank
    const int band = kSplit ? (kTile + sched.splits - 1) / sched.splits : kTile;
    const int band_rows = kSplit ? max(0, min(kTile, (slice_rank + 1) * band) - slice_rank * band) : 0;
    const int m_left = kSplit ? p.M - (first_item % sched.m_tiles) * T : 0;
    const int m_valid = kSplit ? min(T, m_left) : 0;
    // split-K: this CTA's raw sums lie over the (then idle) ring as [group of four tokens][channel], 16 bytes each, so that 32
    // lanes (channels) touch 512 contiguous bytes.  The CTA that finishes a band fetches its channels from all slices.
    // Sent to it by st.async instead (which suits the few rows of the decode kernels), 128 channels x T sums took longer: 200 rows on
    // 3584 -> 3584 14.3 us against 12.9, on 18944 -> 3584 29.9 / 28.3, 96 rows on 3584 -> 4608 12.0 / 11.1.
    constexpr uint32_t group_bytes = kParkedGroupBytes;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kMaxW; ++i) { mbar_init(smem_u32(&bar_wfull[i]), 1); mbar_init(smem_u32(&bar_wempty[i]), kConvWarps / 2); }
        for (int i = 0; i < kMaxX; ++i) { mbar_init(smem_u32(&bar_xfull[i]), 1); mbar_init(smem_u32(&bar_xempty[i]), 1); }
        for (int i = 0; i < kMaxA; ++i) {
            mbar_init(smem_u32(&bar_conv[i]), kConvWarps);
            mbar_init(smem_u32(&bar_empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&bar_tfull[i]), 1); mbar_init(smem_u32(&bar_tempty[i]), 2 * kEpiWarps); }
        mbar_init(smem_u32(&bar_done), 2 * (kConvWarps + kEpiWarps));
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    auto load_weights = [&](uint32_t elected, int item, int kb, int slot) {
        const uint32_t full = smem_u32(&bar_wfull[slot]);
        mbar_expect_tx(elected, full, kWBytes);
        tma_load_2d(elected, wring + slot * kWBytes, &tmap_w, 0, ((2 * (item / sched.m_tiles) + (int)rank) * sched.kblocks + kb) * kTile, full);
    };
    pair_enter();
    const int w_pre = min(kb1 - kb0, nw);              // K blocks of the weight ring's first pass
    if (warp == 2 + kConvWarps + kEpiWarps) {
        const uint32_t el = elect_one();
        for (int i = 0; i < w_pre; ++i) load_weights(el, first_item, kb0 + i, i);
    }
    const uint32_t tmem_base = pair_tmem_begin(warp, &s_tmem_base, kTmemCols);
    pdl_launch_dependents();

    if (warp == 0) {
        // ================= activation producer (both CTAs) =================
        const uint32_t el = elect_one();
        pdl_wait();
        int slot = 0;
        uint32_t phase = 1;                                // parity that a free slot shows on its first use
        bool ok = true;
        for (int item = first_item; item < items && ok; item += item_step) {
            const int row0 = (item % sched.m_tiles) * T + (int)rank * half;
            for (int kb = kb0; kb < kb1; ++kb) {
                ok = !s_abort && warp_wait(smem_u32(&bar_xempty[slot]), phase, p.status, kDevTimeoutEmpty);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; s_abort = 1; break; }
                const uint32_t xfull_local = smem_u32(&bar_xfull[slot]);
                mbar_expect_tx(leader ? el : 0u, xfull_local, 2 * x_bytes);
                const uint32_t xfull = map_to_cta(xfull_local, leader_cta);
                const uint32_t xs = smem_base + slot * x_bytes;
                tma_load_2d_pair(el, xs, &tmap_x, kb * kKB, row0, xfull);
                tma_load_2d_pair(el, xs + xhalf_bytes, &tmap_x, kb * kKB + 64, row0, xfull);
                if (++slot == nx) { slot = 0; phase ^= 1; }
            }
        }
        if (!ok) {
            const long long t0 = clock64();                // let copies that are still in flight land
            while (clock64() - t0 < 2000000) {}
        }
    } else if (warp == 1) {
        // ================= MMA issuer (leader CTA only) =================
        if (leader) {
            const uint32_t el = elect_one();
            const uint32_t idesc = make_idesc_mn(2 * kTile, T, 1, 1);          // A, B = bf16
            const uint16_t both = (uint16_t)(3u << crank);                      // this CTA and its partner
            int tl = 0, xslot = 0, aslot = 0;
            uint32_t xphase = 0, aphase = 0;
            bool ok = true;
            for (int item = first_item; item < items && ok; item += item_step, ++tl) {
                const int as = acc_stages == 2 ? (tl & 1) : 0;
                const uint32_t aph = acc_stages == 2 ? ((tl >> 1) & 1) : (tl & 1);
                ok = __all_sync(0xffffffffu, !s_abort && mbar_wait<true>(smem_u32(&bar_tempty[as]), aph ^ 1, p.status, kDevTimeoutTmemEmpty));
                if (!ok) { s_abort = 1; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * T;
                for (int kb = kb0; kb < kb1; ++kb) {
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_xfull[xslot]), xphase, p.status, kDevTimeoutFull) &&
                                                     mbar_wait<true>(smem_u32(&bar_conv[aslot]), aphase, p.status, kDevTimeoutFull));
                    if (!ok) { s_abort = 1; break; }
                    tc_fence_after();
                    const uint32_t xs = smem_base + xslot * x_bytes;
                    const uint32_t a_t = tmem_base + a_col0 + aslot * kACols;
#pragma unroll
                    for (int k = 0; k < kKB / 16; ++k) {
                        // K = 16 bf16 per MMA: 8 TMEM columns of A, 32 bytes inside the 128-byte swizzle span of B
                        const uint64_t db = make_smem_desc(xs + (k >> 2) * xhalf_bytes) + 2 * (k & 3);
                        umma_f16_ts_pair(el, d_tmem, a_t + k * 8, db, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit_both(el, smem_u32(&bar_xempty[xslot]), both);
                    umma_commit_both(el, smem_u32(&bar_empty[aslot]), both);
                    if (++aslot == n_a) { aslot = 0; aphase ^= 1; }
                    if (++xslot == nx) { xslot = 0; xphase ^= 1; }
                }
                if (ok) umma_commit_both(el, smem_u32(&bar_tfull[as]), both);
            }
        }
        if (!kSplit) pair_tmem_release(smem_u32(&bar_done), tmem_base, kTmemCols, p.status);
    } else if (warp == 2 + kConvWarps + kEpiWarps) {
        // ================= weight producer (both CTAs) =================
        // Its own thread: the weights do not depend on the predecessor, and a slot is refilled as soon as its tile has been
        // widened, up to n_a blocks ahead of the tensor core.
        const uint32_t el = elect_one();
        int slot = w_pre == nw ? 0 : w_pre;
        uint32_t phase = w_pre == nw ? 0 : 1;
        bool ok = true;
        for (int item = first_item; item < items && ok; item += item_step) {
            for (int kb = item == first_item ? kb0 + w_pre : kb0; kb < kb1; ++kb) {
                ok = !s_abort && warp_wait(smem_u32(&bar_wempty[slot]), phase, p.status, kDevTimeoutEmpty);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; s_abort = 1; break; }
                load_weights(el, item, kb, slot);
                if (++slot == nw) { slot = 0; phase ^= 1; }
            }
        }
        if (!ok) {
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
    } else if (warp < 2 + kConvWarps) {
        // ================= converters (warps 2..9 of both CTAs) =================
        // Two teams of four warps take turns (a lane widens a whole row), so that one team's waits and TMEM stores hide under
        // the other's arithmetic, which is what bounds the pair of them.
        const int team = (warp - 2) >> 2;
        const int q = warp & 3;                           // TMEM lane quarter this warp may write
        const int row = q * 32 + lane;                    // weight row (channel) of this lane
        const uint32_t swizzle = (uint32_t)(row & 7);
        const uint32_t dst0 = tmem_base + a_col0 + ((uint32_t)(q * 32) << 16);
        const uint32_t conv0 = map_to_cta(smem_u32(&bar_conv[0]), leader_cta);
        int wslot = 0, aslot = 0, turn = 0;
        uint32_t wphase = 0, aphase = 1;                  // (a free TMEM slot shows parity 1 on its first use)
        bool ok = true;
        for (int item = first_item; item < items && ok; item += item_step) {
            for (int kb = kb0; kb < kb1; ++kb, turn ^= 1) {
                if (turn == team) {
                    // First the TMEM slot: its barrier says that the MMAs of block i - n_a are done, hence that block i - nw
                    // (nw >= n_a), whose ring slot this block's codes arrive in, has been widened -- perhaps by the other
                    // team -- and the parity of the slot's `full` barrier is unambiguous.
                    if (s_abort || !mbar_wait(smem_u32(&bar_empty[aslot]), aphase, p.status, kDevTimeoutEmpty) ||
                        !mbar_wait(smem_u32(&bar_wfull[wslot]), wphase, p.status, kDevTimeoutFull)) { s_abort = 1; ok = false; break; }
                    tc_fence_after();
                    const uint32_t row_addr = wring + wslot * kWBytes + row * 128;
                    uint32_t v[32];
                    widen_half_row(row_addr, swizzle, 0, v);
                    __syncwarp();
                    tmem_st32(dst0 + aslot * kACols, v);
                    widen_half_row(row_addr, swizzle, 1, v);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&bar_wempty[wslot]));        // the codes are in registers
                    tmem_st32(dst0 + aslot * kACols + 32, v);
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(conv0 + (uint32_t)(aslot * sizeof(uint64_t)));
                }
                if (++wslot == nw) { wslot = 0; wphase ^= 1; }
                if (++aslot == n_a) { aslot = 0; aphase ^= 1; }
            }
        }
        pair_tmem_done(smem_u32(&bar_done), leader_cta, lane);
    } else {
        // ================= epilogue (warps 10..17 of both CTAs) =================
        pdl_wait();                                        // y may still be in use by the predecessor
        const int q = warp & 3;
        const int h = (warp - 2 - kConvWarps) >> 2;        // which half of the tile's tokens
        const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16) + h * half;
        const bool odd = lane & 1;
        int tl = 0;
        bool ok = true;
        for (int item = first_item; item < items && ok; item += item_step, ++tl) {
            const int as = acc_stages == 2 ? (tl & 1) : 0;
            const uint32_t aph = acc_stages == 2 ? ((tl >> 1) & 1) : (tl & 1);
            const int n = (2 * (item / sched.m_tiles) + (int)rank) * kTile + q * 32 + lane;
            const int m0 = (item % sched.m_tiles) * T + h * half;
            float ws = 0.f, bs = 0.f;
            if (!kSplit && n < p.N) {
                ws = ld_dep(p.w_scale + n);
                if (p.bias) bs = ld_dep(p.bias + n);
            }
            if (!mbar_wait(smem_u32(&bar_tfull[as]), aph, p.status, kDevTimeoutTmemFull)) { s_abort = 1; ok = false; break; }
            tc_fence_after();
            if constexpr (!kSplit) {
                // All sums leave tensor memory as bf16 pairs of tokens before the first is stored: with one accumulator stage the
                // next tile's MMAs wait for that, and behind the stores they did for 8000 SM cycles of a tile's 33000 at T = 224 (3584 -> 37888
                // 200 rows 47.3 -> 45.4 us, four 7B projections of 4096 rows 1540 -> 1461).  Then a lane stores two channels of one token: even lanes the even tokens,
                // odd lanes the odd ones.
                __nv_bfloat16* yp = p.y + (size_t)m0 * p.ldy + (n & ~1) + (odd ? p.ldy : 0);
                const bool in = (n & ~1) < p.N;                // (N is even)
                uint32_t o[64];
#pragma unroll
                for (int c = 0; c < 128; c += 16) {
                    if (c < half) {
                        uint32_t v[16];
                        __syncwarp();
                        tmem_ld16_nowait(t_lane + as * T + c, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; j += 2) o[(c + j) / 2] = pack_bf16x2(fmaf(__uint_as_float(v[j]), ws, bs), fmaf(__uint_as_float(v[j + 1]), ws, bs));
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(&bar_tempty[as]), leader_cta));
                const uint32_t sel = odd ? 0x3276u : 0x5410u;
#pragma unroll
                for (int c = 0; c < 128; c += 16) {
                    if (c < half) {
#pragma unroll
                        for (int j = 0; j < 16; j += 2) {
                            const uint32_t own = o[(c + j) / 2], other = __shfl_xor_sync(0xffffffffu, own, 1);
                            if (in && m0 + c + j + (odd ? 1 : 0) < p.M) *reinterpret_cast<uint32_t*>(yp + (size_t)(c + j) * p.ldy) = __byte_perm(own, other, sel);
                        }
                    }
                }
            } else {
                // the pair's MMAs are done, so this CTA's ring is free
                const uint32_t dst = smem_base + (uint32_t)(h * half >> 2) * group_bytes + (uint32_t)(q * 32 + lane) * 16u;
                for (int c = 0; c < half; c += 32) {
                    uint32_t v[32];
                    __syncwarp();
                    tmem_ld16_nowait(t_lane + c, v);
                    if (c + 16 < half) tmem_ld16_nowait(t_lane + c + 16, v + 16);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        if (j == 16 && c + 16 >= half) break;
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (uint32_t)((c + j) >> 2) * group_bytes), "r"(v[j]), "r"(v[j + 1]),
                                     "r"(v[j + 2]), "r"(v[j + 3]) : "memory");
                    }
                }
            }
        }
        pair_tmem_done(smem_u32(&bar_done), leader_cta, lane);
    }

    if constexpr (kSplit) {
        // ---- this CTA finishes its band: slices added in rank order, scaled, stored ----
        __syncwarp();
        pdl_wait();
        cluster_sync_all();                                // every CTA's sums are parked
        if (warp == 1) pair_tmem_release(smem_u32(&bar_done), tmem_base, kTmemCols, p.status);
        if (!s_abort) {
            finish_parked_band(p, smem_base, sched.splits, (int)rank, slice_rank * band, band_rows, m_valid,
                               (2 * (first_item / sched.m_tiles) + (int)rank) * kTile, (first_item % sched.m_tiles) * T, 1.f, 1.f, kThreads);
        }
    }

    pair_leave();
}

bool encode_x_tokens(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes, uint32_t box_rows) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {pitch_bytes};
    cuuint32_t box[2] = {64u, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool kSplit>
cudaError_t launch_kernel(const W8a16PairPlan& pl, const UmmaArgs& a, const CUtensorMap& tw, const CUtensorMap& tx, cudaStream_t stream) {
    auto kern = w8a16_pair_kernel<kSplit>;
    static SmemOptIn opted;
    cudaError_t e = ensure_dynamic_smem((const void*)kern, kSmemBytes, opted);
    if (e != cudaSuccess) return e;
    PairSched16 s;
    s.n_tiles = pl.n_tiles; s.m_tiles = pl.m_tiles; s.tokens = pl.tokens; s.splits = pl.splits;
    s.kblocks = (a.K + kKB - 1) / kKB; s.kblocks_per_split = pl.kblocks_per_split;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)pl.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
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
    return counted(cudaLaunchKernelEx(&cfg, kern, tw, tx, a, s));
}

}  // namespace

// Tokens per tile and K slices: the cheapest by a model of the kernel, microseconds, fitted to back-to-back calls with every
// (T, slices) on twelve layer shapes (1280 -> 1536 .. 2048 -> 11008 .. 18944 -> 3584, 3584 -> 37888) at 40 to 1031 rows; the choice is
// 0.7 % slower than the best of the sweep on average.  A K block takes the longer of the weights' way (ring, widening, HBM:
// 0.45, a little more when every SM streams) and the tensor core's (0.19 + 0.0016 T), and all blocks together what the
// power limit allows (0.17 + 0.0025 T per pair and block: large calls run at 1.2 GHz).  A call starts later the more SMs it
// needs at once; a tile adds its epilogue; slices add the hand-over of T x (1 - 1/s) sums per channel and what a cluster
// takes to start (slices are only taken when all clusters fit at once: a second wave never paid).
W8a16PairPlan plan_w8a16_pair(int64_t M, int64_t K, int64_t N, int force_tokens, int force_splits) {
    W8a16PairPlan best{};
    const int kblocks = (int)((K + kKB - 1) / kKB);
    const int n_tiles = (int)((N + 255) / 256);
    static const double cluster_start[5] = {0, 0, 0.24, 0.22, 1.48};
    double best_cost = 1e30;
    for (int splits = 1; splits <= 4; ++splits) {
        if (force_splits > 0 && splits != (force_splits > 4 ? 4 : force_splits)) continue;
        if (splits > kblocks) break;
        const int kps = (kblocks + splits - 1) / splits;
        if ((kblocks + kps - 1) / kps != splits) continue;                    // would leave an empty slice
        if (force_splits <= 0 && splits > 1 && kps < 4) break;
        const int slots = splits == 1 ? max_active_clusters((const void*)w8a16_pair_kernel<false>, kThreads, kSmemBytes, 2)
                                      : max_active_clusters((const void*)w8a16_pair_kernel<true>, kThreads, kSmemBytes, 2 * splits);
        if (slots < 1) continue;
        for (int tokens = 32; tokens <= 256; tokens += 32) {
            if (force_tokens > 0 && tokens != force_tokens) continue;
            if (force_tokens <= 0 && tokens >= M + 32) break;
            const int m_tiles = (int)((M + tokens - 1) / tokens);
            const long items = (long)n_tiles * m_tiles;
            if (force_splits <= 0 && splits > 1 && items > slots) continue;
            const long rounds = (items + slots - 1) / slots;
            const double load = (double)(items < slots ? items : slots) * 2 * splits / sm_count();
            const double weights = 0.447 * (1 + 0.08 * load), tensor = (0.193 + 0.00163 * tokens) * (1 + 0.023 * load);
            const double t_block = weights > tensor ? weights : tensor;
            const double drain = 0.0149 * tokens;
            const double chain = rounds * kps * t_block + (rounds - 1) * (0.08 + drain);
            const double power = (double)items * splits * kps / (sm_count() / 2) * (0.173 + 0.00246 * tokens);
            const double tail = splits > 1 ? 1.31 + cluster_start[splits] + 0.0303 * tokens * (1.0 - 1.0 / splits) : drain;
            const double cost = (chain > power ? chain : power) + 2.8 * load + tail;
            if (cost < best_cost) {
                best_cost = cost;
                best.n_tiles = n_tiles; best.m_tiles = m_tiles; best.tokens = tokens; best.splits = splits; best.kblocks_per_split = kps;
                best.grid = splits > 1 ? (int)(items * 2 * splits) : 2 * (int)(items < slots ? items : slots);
            }
        }
    }
    return best;
}

cudaError_t launch_w8a16_pair(const W8a16PairPlan& pl, const UmmaArgs& a, const void* x, int64_t ldx, cudaStream_t stream, const char** why) {
    CUtensorMap tw, tx;
    if (pl.tokens < 32 || !encode_u8_2d(&tw, a.w, (uint64_t)(pack_ntiles(a.N) * pack_kblocks(a.K) * 128), 128, kTile) ||
        !encode_x_tokens(&tx, x, (uint64_t)a.M, (uint64_t)a.K, (uint64_t)ldx * 2, (uint32_t)pl.tokens / 2)) {
        if (why) *why = "no plan, or cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    return pl.splits > 1 ? launch_kernel<true>(pl, a, tw, tx, stream) : launch_kernel<false>(pl, a, tw, tx, stream);
}

}  // namespace fp8lin
