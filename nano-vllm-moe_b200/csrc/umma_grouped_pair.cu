// Grouped W8A8 GEMM of prefill-sized expert batches on CTA pairs (tcgen05 cta_group::2), channels as the MMA's M:
//
//   D[256 channels, R rows] = W_e[256 channels, K] . xq[rows of one chunk, K]^T        R = the chunk's rows, rounded up to 32
//
// for every chunk of at most 320 routed rows that share an expert e (even chunks, moe_place_kernel; the rows already e4m3 and in
// sorted order) and every item of 256 channels:
//   gate_up (kDown = false)  an item is gate tile t and up tile t of the expert (128 channels each).  CTA r of the pair takes
//             channels [64 r, 64 r + 64) of BOTH, so that a gate value and its up value meet in one CTA: warps of the gate
//             lanes and of the up lanes swap half of their values through shared memory (gate_up_swap) and write
//             hq[sorted position][channel] = e4m3(h / h_scale), h = bf16(bf16(silu(g)) * u) from g, u rounded to bf16 (the
//             eager two-rounding SiluAndMul of the reference's experts).
//   down    (kDown = true)   an item is channel tiles 2 t and 2 t + 1, one per CTA; out[routed row][channel] =
//             bf16(acc * scale * routing weight).
//
//   warp 0      TMA producer (both CTAs): 16 KB of weights and R/2 rows per K block
//   warp 1      MMA issuer (leader): four tcgen05.mma 256 x N x 32 per K block, twice that where R > 256 (N <= 256 each)
//   warps 2..17 epilogue: warp (q, h) owns TMEM lanes [32 q, 32 q + 32) and every fourth piece of 16 rows
//
// What bounds it: memory and the tensor core about equally at some 270 rows per expert (weights and rows once from memory: 59 us for
// gate_up of 60 experts 2048 -> 2 x 1408, its MMAs 576 SM cycles per K block of 288 rows), memory alone below.  So a chunk holds all
// rows of an expert where it can (its weights come once), rows are the MMA's N (273 rows of an expert on average are multiplied as
// 288, in 128-row tiles as 384), and a K block of 256 channels x 288 rows moves 34 KB into each SM where 128 x 256 tiles move 48 KB
// for a third of the products.  16384 rows of 60 experts, in a loop under the power limit: the block 278 us with 128 x 256 tiles on
// one CTA (umma_grouped_rows.cu), 219 here; 8192 rows 180 / 148; 2048 rows 115 / 105.  Five or six slots of loads in flight: asking
// weights beyond them into L2 in front was slower the further (192 us without, 196 six blocks ahead, 206 sixteen).
//
// Sixteen epilogue warps: eight take longer over an item of gate_up than its MMAs do.
//
// Work: the items of all chunks in a row, chunk after chunk, are dealt out to the pairs, so that those at work at one time share a
// few chunks' rows, which stay in L2 (a stretch of the row per pair, each on chunks of its own: 85 MB more from memory, gate_up of 16384
// rows 99 us against 92).  Where a pair has only a few items, the row is cut into one stretch of equal cost per pair instead,
// between two items or between two groups of 32 rows of an item (both sides then load its weights).
//
// Tensor memory: the items of a pair lie at the two ends of the 512 columns in turn.  Items whose sums do not fit beside each
// other overlap in the middle; the epilogue reads that part first and hands it to the next item's MMAs (bar_tfree) before
// the rest.  All waits are bounded; the epilogue warps vote on each item, because they meet at named barriers.
#include "umma_common.cuh"

namespace fp8lin {

namespace {

constexpr int kEpiWarps = 16;
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr int kKB = 128;
constexpr int kWBytes = 128 * kKB;                 // this CTA's 128 channel rows
constexpr int kMaxSlots = 10;
constexpr int kRingBytes = 204 * 1024;             // 16 KB + 64 R bytes per slot, R = the longest chunk
constexpr int kPiece = 16;                         // rows of an epilogue step
constexpr int kSwapBytes = kPiece * 64;            // bf16 values of a piece x 32 channels, one buffer per warp pair
constexpr int kCodeBytes = kPiece * 32;            // e4m3 of a piece x 32 channels
constexpr int kSmemBytes = kRingBytes + kEpiWarps / 2 * (kSwapBytes + kCodeBytes) + 1024;
constexpr int kTmemCols = 512;
constexpr int kFewItems = 4;                       // fewer work items per pair: one stretch of them each
constexpr int kMinGroups = 3;                      // a cut leaves at least so many groups of 32 rows on both sides
static_assert(kGroupedPairMaxRows <= 320 && (kWBytes + 64 * kGroupedPairMaxRows) * 5 <= kRingBytes, "five slots at least");

// The work of one pair: items w0, w0 + step, .. (n of them; item w is channel item w % n_items of chunk w / n_items), without the
// first k0 groups of 32 rows of the first one and, unless k1 is 0, of the last one only the first k1 groups.
struct Stretch {
    int w0, step, n, k0, k1;
};

// One work item as every role sees it (values uniform over the warp): up to `cols` rows, in one or two MMA tiles of n_a and n_b.
struct Item {
    int expert, t, start, rows, cols, n_a, n_b;
};
__device__ __forceinline__ Item load_item(const int4* chunks, int n_items, const Stretch& s, int i) {
    const int w = s.w0 + i * s.step;
    const int* v = reinterpret_cast<const int*>(chunks + w / n_items);
    Item r;
    r.t = w % n_items;
    r.expert = uniform(ld_dep(v));
    const int rows = uniform(ld_dep(v + 2));
    const int from = i == 0 ? 32 * s.k0 : 0, to = i == s.n - 1 && s.k1 ? min(rows, 32 * s.k1) : rows;
    r.start = uniform(ld_dep(v + 1)) + from;
    r.rows = to - from;
    r.cols = (r.rows + 31) & ~31;
    r.n_a = r.cols <= 256 ? r.cols : ((r.cols >> 1) + 31) & ~31;
    r.n_b = r.cols - r.n_a;
    return r;
}

// Boxes of the weights (64 rows for a half of gate_up, 128 for down; 16 for up rows inside tiles) and of 16, 32, .. 128 routed
// rows: a K block is two to four TMA instructions.
struct GroupedPairMaps {
    CUtensorMap w, w16, x[8];
};

template <bool kDown>
__global__ void __launch_bounds__(kThreads, 1)
grouped_pair_kernel(const __grid_constant__ GroupedPairMaps maps, GroupedArgs p, int slot_bytes, int n_slots) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kMaxSlots];       // leader's: both CTAs' bytes
    __shared__ __align__(8) uint64_t bar_empty[kMaxSlots];      // the MMAs that read the slot are done (both CTAs')
    __shared__ __align__(8) uint64_t bar_tfull[2];
    __shared__ __align__(8) uint64_t bar_tfree[2];              // leader's: item i's columns that item i + 1 takes have been read
    __shared__ __align__(8) uint64_t bar_done;                  // tensor memory of both CTAs has been read for the last time
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile int s_abort;
    __shared__ __align__(16) int s_routed[2][kDown ? kGroupedPairMaxRows : 4];
    __shared__ __align__(16) float s_rw[2][kDown ? kGroupedPairMaxRows : 4];
    __shared__ int2 s_ends[2];

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kMaxSlots; ++i) { mbar_init(smem_u32(&bar_full[i]), 1); mbar_init(smem_u32(&bar_empty[i]), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&bar_tfull[i]), 1); mbar_init(smem_u32(&bar_tfree[i]), 2 * kEpiWarps); }
        mbar_init(smem_u32(&bar_done), 2 * kEpiWarps);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    pair_enter();
    const uint32_t tmem_base(pair_tmem_begin(warp, &s_tmem_base, kTmemCols));
    pdl_launch_dependents();
    pdl_wait();                    // the chunk list, the rows and the outputs all come from predecessors

    const int n_items = p.n_tiles;                    // channel items per chunk (set by the launcher)
    const int KB = p.kblocks;
    const int n_chunks = uniform(ld_dep(p.meta));
    const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    Stretch my{pair, pairs, (n_chunks * n_items - pair + pairs - 1) / pairs, 0, 0};
    if (n_chunks * n_items < kFewItems * pairs) {
        // All threads look for the chunks that the two ends of this pair's stretch lie in (a chunk's .w is the cost of all in front).
        const int64_t cost = (int64_t)ld_dep(p.meta + 2) * n_items;
        const int64_t end0 = cost * pair / pairs, end1 = cost * (pair + 1) / pairs;
        int c0 = 0, c1 = 0;                           // chunks that begin at or in front of the ends
        for (int c = 0; c < n_chunks; c += kThreads) {
            const int i = c + (int)threadIdx.x;
            const int64_t at = i < n_chunks ? (int64_t)ld_dep(reinterpret_cast<const int*>(p.chunks + i) + 3) * n_items : INT64_MAX;
            c0 += __syncthreads_count(at <= end0);
            c1 += __syncthreads_count(at <= end1);
        }
        if (threadIdx.x < 2) {
            int w = 0, k = 0;
            if (n_chunks > 0) {
                const int c = (threadIdx.x ? c1 : c0) - 1;
                const int* v = reinterpret_cast<const int*>(p.chunks + c);
                const int groups = (ld_dep(v + 2) + 31) >> 5, item_cost = grouped_pair_cost(groups);
                const int at = (int)((threadIdx.x ? end1 : end0) - (int64_t)ld_dep(v + 3) * n_items);
                w = at / item_cost;
                k = ((at - w * item_cost) * groups + item_cost / 2) / item_cost;
                if (k < kMinGroups || k > groups - kMinGroups) k = 2 * k < groups ? 0 : groups;
                w += c * n_items;
                if (k == groups) { ++w; k = 0; }
            }
            s_ends[threadIdx.x] = make_int2(w, k);
        }
        __syncthreads();
        const int2 a = s_ends[0], b = s_ends[1];
        my.w0 = uniform(a.x); my.step = 1; my.k0 = uniform(a.y); my.k1 = uniform(b.y);
        my.n = uniform(b.x - a.x + (b.y > (a.x == b.x ? a.y : 0) ? 1 : 0));
    }

    if (warp == 0) {
        // ================= TMA producer (both CTAs) =================
        const uint32_t el = elect_one();
        int st = 0;
        uint32_t phase = 1;                           // parity that a free slot shows on its first use
        bool ok = true;
        // packed weight rows of an item's K block 0: gate_up 64 rows each of gate tile t and up tile t; down its own tile (the last
        // item of an odd number of tiles has none for CTA 1: it multiplies tile 2 t again and stores nothing)
        struct WeightRows {
            int a, up[4];
        };
        // up channels start at row N of the expert's weight, perhaps inside a tile: then four boxes of 16 rows, which a tile boundary
        // (N is a multiple of 16) never cuts
        const bool up_whole = (p.N & 63) == 0;
        auto weight_rows = [&](const Item& ch) {
            WeightRows r;
            const int tile = kDown ? min(2 * ch.t + (int)rank, p.w_tiles - 1) : ch.t;
            r.a = (ch.expert * p.w_tiles + tile) * KB * 128 + (kDown ? 0 : (int)rank * 64);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                // (channels beyond the last exist in no tile and are not stored)
                const int up = min(p.N + ch.t * 128 + (int)rank * 64 + 16 * i, p.w_tiles * 128 - 16);
                r.up[i] = (ch.expert * p.w_tiles + (up >> 7)) * KB * 128 + (up & 127);
            }
            return r;
        };
        for (int i = 0; i < my.n && ok; ++i) {
            const Item ch = load_item(p.chunks, n_items, my, i);
            const WeightRows wr = weight_rows(ch);
            // this CTA's half of either MMA tile's rows
            const int half_a = ch.n_a >> 1, half_b = ch.n_b >> 1;
            const int row_a = ch.start + (int)rank * half_a, row_b = ch.start + ch.n_a + (int)rank * half_b;
            const CUtensorMap* map_a = &maps.x[(half_a >> 4) - 1];
            const CUtensorMap* map_b = &maps.x[half_b ? (half_b >> 4) - 1 : 0];
            const uint32_t bytes = (uint32_t)(kWBytes + (ch.cols >> 1) * kKB);
            for (int kb = 0; kb < KB; ++kb) {
                ok = !s_abort && warp_wait(smem_u32(&bar_empty[st]), phase, p.status, kDevTimeoutEmpty);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; s_abort = 1; break; }
                const uint32_t full_local = smem_u32(&bar_full[st]);
                mbar_expect_tx(leader ? el : 0u, full_local, 2 * bytes);
                const uint32_t full = map_to_cta(full_local, 0);
                const uint32_t sa = smem_base + (uint32_t)(st * slot_bytes);
                tma_load_2d_pair(el, sa, &maps.w, 0, wr.a + kb * 128, full);
                if (!kDown) {
                    if (up_whole) tma_load_2d_pair(el, sa + kWBytes / 2, &maps.w, 0, wr.up[0] + kb * 128, full);
                    else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) tma_load_2d_pair(el, sa + kWBytes / 2 + j * 2048, &maps.w16, 0, wr.up[j] + kb * 128, full);
                    }
                }
                tma_load_2d_pair(el, sa + kWBytes, map_a, kb * kKB, row_a, full);
                if (half_b) tma_load_2d_pair(el, sa + kWBytes + half_a * kKB, map_b, kb * kKB, row_b, full);
                if (++st == n_slots) { st = 0; phase ^= 1; }
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
            int st = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tl = 0; tl < my.n && ok; ++tl) {
                const Item ch = load_item(p.chunks, n_items, my, tl);
                const uint32_t idesc_a = make_idesc_mn(256, ch.n_a, 0, 0), idesc_b = make_idesc_mn(256, ch.n_b, 0, 0);
                if (tl > 0) {                         // what item tl - 1 has in these columns has been read
                    const int prev = tl - 1;
                    ok = __all_sync(0xffffffffu, !s_abort && mbar_wait<true>(smem_u32(&bar_tfree[prev & 1]), (prev >> 1) & 1, p.status, kDevTimeoutTmemEmpty));
                    if (!ok) { s_abort = 1; break; }
                }
                tc_fence_after();
                const uint32_t d_a = tmem_base + ((tl & 1) ? kTmemCols - ch.cols : 0), d_b = d_a + ch.n_a;
                for (int kb = 0; kb < KB; ++kb) {
                    ok = __all_sync(0xffffffffu, !s_abort && mbar_wait(smem_u32(&bar_full[st]), phase, p.status, kDevTimeoutFull));
                    if (!ok) { s_abort = 1; break; }
                    tc_fence_after();
                    const uint32_t sa = smem_base + (uint32_t)(st * slot_bytes);
                    const uint64_t dw = make_smem_desc(sa);
                    const uint64_t dx = make_smem_desc(sa + kWBytes);
#pragma unroll
                    for (int k = 0; k < kKB / 32; ++k) umma_f8_pair(el, d_a, dw + 2 * k, dx + 2 * k, idesc_a, (kb > 0 || k > 0) ? 1u : 0u);
                    if (ch.n_b) {
                        const uint64_t dy = make_smem_desc(sa + kWBytes + (ch.n_a >> 1) * kKB);
#pragma unroll
                        for (int k = 0; k < kKB / 32; ++k) umma_f8_pair(el, d_b, dw + 2 * k, dy + 2 * k, idesc_b, (kb > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit_both(el, smem_u32(&bar_empty[st]), both);
                    if (++st == n_slots) { st = 0; phase ^= 1; }
                }
                if (ok) umma_commit_both(el, smem_u32(&bar_tfull[tl & 1]), both);
            }
        }
        pair_tmem_release(smem_u32(&bar_done), tmem_base, kTmemCols, p.status);
    } else {
        // ================= epilogue (warps 2..17 of both CTAs) =================
        const int q = warp & 3;                       // TMEM lane quarter
        const int h = (warp - 2) >> 2;                // takes pieces h, h + 4, ..
        const int et = threadIdx.x - 64;              // 0..511 among the epilogue threads
        const float in_scale = fmaxf(ld_dep(p.input_scale), 1e-12f);
        const ExactDiv div_h(kDown ? 1.f : fmaxf(ld_dep(p.h_scale), 1e-12f));
        const bool up = q >= 2;                       // gate_up: lanes of quarters 2, 3 are up channels
        const int pair = (q & 1) + 2 * h;             // the warps of quarters q and q ^ 2 share 32 channels and a buffer
        const uint32_t swap_buf = smem_base + kRingBytes + pair * (kSwapBytes + kCodeBytes);
        const uint32_t code_buf = swap_buf + kSwapBytes;
        const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
        // output channel of this lane (gate_up: of the pair of values) and its multiplier
        auto channel_of = [&](int t) { return kDown ? (2 * t + (int)rank) * 128 + q * 32 + lane : t * 128 + (int)rank * 64 + (q & 1) * 32 + lane; };
        auto scale_of = [&](int e, int n) -> float {
            if (n >= p.N) return 0.f;
            return in_scale * ld_dep(p.w_scale + (kDown ? (size_t)e * p.N + n : (size_t)e * 2 * p.N + (up ? p.N : 0) + n));
        };
        // of the next item: this lane's multiplier; down: the routed row that this thread puts into shared memory
        int next_routed = 0;
        float next_rw = 0.f, next_scale = 0.f;
        Item next{};
        auto prefetch = [&](int i) {
            next = load_item(p.chunks, n_items, my, i);
            next_scale = scale_of(next.expert, channel_of(next.t));
            if (kDown && et < next.rows) {
                next_routed = ld_dep(p.sorted_rows + next.start + et);
                next_rw = ld_dep(p.topk_w + next_routed);
            }
        };
        if (my.n > 0) prefetch(0);
        for (int tl = 0; tl < my.n; ++tl) {
            const Item ch = next;
            const int n = channel_of(ch.t);
            const float scale = next_scale;
            const int side = tl & 1;
            // (the readers of this buffer's last contents passed the vote of the item before)
            int* const routed = s_routed[side];
            float* const row_w = s_rw[side];
            if (kDown && et < ch.cols) { routed[et] = next_routed; row_w[et] = next_rw; }
            next.cols = 0;
            if (tl + 1 < my.n) prefetch(tl + 1);
            // pieces from the middle outwards: the first `shared` of them lie where the next item begins
            const int pieces = ch.cols / kPiece;
            const int shared = max(0, ch.cols + next.cols - kTmemCols) / kPiece;
            const uint32_t free_bar = map_to_cta(smem_u32(&bar_tfree[side]), 0);
            if (shared <= h) {                            // none of them this warp's, and it has read all of the item before
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(free_bar);
            }
            const bool arrived = mbar_wait(smem_u32(&bar_tfull[side]), (tl >> 1) & 1, p.status, kDevTimeoutTmemFull);
            if (named_sync_any(9, kEpiWarps * 32, !arrived)) { s_abort = 1; break; }
            tc_fence_after();
            for (int i = h; i < pieces; i += kEpiWarps / 4) {
                const int m0 = side ? kPiece * i : ch.cols - kPiece * (i + 1);    // first row (of the item) of the piece
                const uint32_t t_piece = t_lane + (side ? kTmemCols - ch.cols : 0) + m0;
                auto release = [&]() {
                    if (i < shared && i + kEpiWarps / 4 >= shared) {                          // the last of the shared pieces is in registers
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_remote(free_bar);
                    }
                };
                uint32_t v[kPiece];
                __syncwarp();
                tmem_ld16_nowait(t_piece, v);
                tmem_ld_wait();
                release();
                if constexpr (kDown) {
                    // Two lanes swap halves: an even lane stores two channels of the even rows, an odd lane of the odd rows.
                    const bool odd = lane & 1;
                    const bool in = (n & ~1) < p.N;
                    __nv_bfloat16* const out = p.out + (n & ~1);
                    const int left = ch.rows - m0 - (odd ? 1 : 0);                // row j (+ 1) of the piece exists for j < left
#pragma unroll
                    for (int j = 0; j < kPiece; j += 4) {
                        const float4 rw = *reinterpret_cast<const float4*>(row_w + m0 + j);
                        const int4 rr = *reinterpret_cast<const int4*>(routed + m0 + j);
                        const uint32_t own0 = pack_bf16x2(__uint_as_float(v[j]) * scale * rw.x, __uint_as_float(v[j + 1]) * scale * rw.y);
                        const uint32_t own1 = pack_bf16x2(__uint_as_float(v[j + 2]) * scale * rw.z, __uint_as_float(v[j + 3]) * scale * rw.w);
                        const uint32_t other0 = __shfl_xor_sync(0xffffffffu, own0, 1), other1 = __shfl_xor_sync(0xffffffffu, own1, 1);
                        const uint32_t sel = odd ? 0x3276u : 0x5410u;
                        if (in && j < left) *reinterpret_cast<uint32_t*>(out + (size_t)(odd ? rr.y : rr.x) * p.ld_out) = __byte_perm(own0, other0, sel);
                        if (in && j + 2 < left) *reinterpret_cast<uint32_t*>(out + (size_t)(odd ? rr.w : rr.z) * p.ld_out) = __byte_perm(own1, other1, sel);
                    }
                } else {
                    uint32_t lo[kPiece / 4], hi[kPiece / 4];              // as the bf16 gate_up row
#pragma unroll
                    for (int j = 0; j < kPiece / 4; ++j) {
                        lo[j] = pack_bf16x2(__uint_as_float(v[2 * j]) * scale, __uint_as_float(v[2 * j + 1]) * scale);
                        hi[j] = pack_bf16x2(__uint_as_float(v[kPiece / 2 + 2 * j]) * scale, __uint_as_float(v[kPiece / 2 + 2 * j + 1]) * scale);
                    }
                    gate_up_swap<kPiece, true>(lo, hi, up, swap_buf, code_buf, 1 + pair, lane, div_h);
                    // 32 bytes per row: thread r of the 64 stores a quarter of a row (N is a multiple of 16)
                    const int r = (up ? 32 : 0) + lane, m = m0 + (r >> 2), nh = (n - lane) + (r & 3) * 8;
                    if (m < ch.rows && nh < p.N)
                        *reinterpret_cast<float2*>(p.hq + (size_t)(ch.start + m) * p.N + nh) = ld_shared_f2(code_buf + (r >> 2) * 32 + (r & 3) * 8);
                }
            }
        }
        pair_tmem_done(smem_u32(&bar_done), 0, lane);
    }

    pair_leave();
}

template <bool kDown>
cudaError_t launch_kernel(const GroupedArgs& a, const GroupedPairMaps& maps, int max_rows, cudaStream_t stream, const char** why) {
    auto kern = grouped_pair_kernel<kDown>;
    static SmemOptIn opted;
    cudaError_t e = ensure_dynamic_smem((const void*)kern, kSmemBytes, opted);
    if (e != cudaSuccess) return e;
    const int pairs = max_active_clusters((const void*)kern, kThreads, kSmemBytes, 2);
    if (pairs < 1) {
        if (why) *why = "no CTA pair fits on this device";
        return cudaErrorInvalidConfiguration;
    }
    const int slot_bytes = kWBytes + 64 * max_rows;
    int n_slots = kRingBytes / slot_bytes;
    if (n_slots > kMaxSlots) n_slots = kMaxSlots;
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
    return counted(cudaLaunchKernelEx(&cfg, kern, maps, a, slot_bytes, n_slots));
}

}  // namespace

cudaError_t launch_grouped_pair_w8a8(GroupedArgs a, int max_rows, const void* w_packed, int num_experts, const void* xq_sorted, int64_t xq_rows,
                                     cudaStream_t stream, const char** why) {
    const bool gate_up = a.hq != nullptr;                          // a.N = I gate channels; the expert's weight holds 2 I channels
    const int tiles = (int)pack_ntiles(a.N);
    a.w_tiles = (int)pack_ntiles(gate_up ? 2 * (int64_t)a.N : a.N);
    a.kblocks = (int)pack_kblocks(a.K);
    a.n_tiles = gate_up ? tiles : (tiles + 1) / 2;
    if (a.N % 16 != 0 || (!gate_up && a.ld_out % 2 != 0) || max_rows < 32 || max_rows > kGroupedPairMaxRows || max_rows % 32 != 0) {
        if (why) *why = "grouped GEMM on CTA pairs: the output width must be a multiple of 16, the chunk size one of 32";
        return cudaErrorInvalidValue;
    }
    GroupedPairMaps maps;
    const uint64_t w_rows = (uint64_t)num_experts * a.w_tiles * a.kblocks * 128;
    bool ok = encode_u8_2d(&maps.w, w_packed, w_rows, 128, gate_up ? 64 : 128);
    // (a map costs the host 0.1 us: only what the kernel reads.  Up rows inside a tile; halves of an MMA tile of up to max_rows, 256 at most)
    maps.w16 = maps.w;
    if (ok && gate_up && (a.N & 63) != 0) ok = encode_u8_2d(&maps.w16, w_packed, w_rows, 128, 16);
    const int boxes = max_rows <= 256 ? max_rows / 32 : 8;
    for (int i = 0; i < boxes && ok; ++i) ok = encode_u8_2d(&maps.x[i], xq_sorted, (uint64_t)xq_rows, (uint64_t)a.K, 16 * (i + 1));
    for (int i = boxes; i < 8; ++i) maps.x[i] = maps.w;
    if (!ok) {
        if (why) *why = "cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    return gate_up ? launch_kernel<false>(a, maps, max_rows, stream, why) : launch_kernel<true>(a, maps, max_rows, stream, why);
}

}  // namespace fp8lin
