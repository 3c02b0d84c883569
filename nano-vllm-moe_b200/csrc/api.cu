// extern "C" surface of libfp8lin.so (declared in include/fp8lin.h).
#include <math.h>
#include <stdarg.h>
#include <atomic>
#include <stdio.h>
#include <string.h>

#include "common.cuh"
#include "kernels.h"

using namespace fp8lin;

namespace {

thread_local char g_err[256] = "";

int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

struct Tuning {
    int stream_splits = -1;   // force split-K factor of the streaming kernel
    int stream_max_m = -1;    // largest M routed to the streaming kernel (W8A8)
    int umma_bn = -1;         // force tile width of the tcgen05 kernel
    int umma_splits = -1;     // force split-K factor of the tcgen05 kernel
    int swap_splits = -1;     // force split-K factor of the swapped-operand decode kernel
    int swap_enable = -1;     // 0 routes decode-sized W8A8 to the mma.sync streaming kernel instead
    int swap_min_m = -1;      // smallest M routed to the swapped-operand kernel
    int swap_preq_min_m = -1; // smallest M for which that kernel takes pre-quantised activations
    int w8a16_swap_enable = -1; // 0 keeps W8A16 on the mma.sync streaming kernel for every M
    int w8a16_swap_min_m = -1;
    int w8a16_umma_min_m = -1;  // smallest M for the dequantise-to-f16 + tcgen05 GEMM route (0 = never)
    int w8a16_chunk_mb = -1;    // size of the f16 weight chunk that route keeps in L2
    int w8a16_pair = -1;        // 0 = never the CTA-pair kernel that widens weights into TMEM, 1 = for every M
    int w8a16_pair_tokens = -1; // force its tokens per tile / its K slices
    int w8a16_pair_splits = -1;
    int w8a8_pair = -1;         // 0 = never the CTA-pair kernel with the rows as the MMA's N, 1 = for every M
    int w8a8_pair_tokens = -1;  // force its tokens per tile / its K slices / whether a cluster takes them (1 = no)
    int w8a8_pair_slices = -1;
    int w8a8_pair_splits = -1;
    int umma_pair = -1;         // 1 = large-M GEMMs on CTA pairs (256 x 256 tiles), 0 = never
    int fuse_quant = -1;        // large-M W8A8: <= 0 (default) = quantise x in a separate pass; 1 = the pass takes the rows
                                // of the first round of tiles, the GEMM's own quantiser warps the rest; n > 1 = the pass
                                // takes the first n rows (rounded up to 128)
    int moe_pair = -1;          // 0 = prefill-sized expert batches never on CTA pairs; 32..320 = always, with chunks of at most so many rows
    int moe_rows_major = -1;    // 0 = prefill-sized expert batches stay on the channel-major grouped kernel
    int mlp_decode_fused = -1;  // 1 = the fused MLP on up to 16 pre-quantised rows computes silu * up in the gate_up kernel (study knob)
    int moe_fused = -1;         // 0 = the expert FFN keeps its separate silu-multiply-quantise pass for every batch size
    int quant_lead = -1;        // row blocks the in-kernel quantiser may run ahead (default: from the tile schedule)
} g_tune;

constexpr int kDefaultStreamMaxM = 64;

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int check_arch() {
    static int cached = -1;
    if (cached >= 0) return cached;
    int dev = 0;
    cudaDeviceProp prop;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return cached = 0;
    return cached = (prop.major == 10) ? 1 : 0;
}

int validate_common(const void* x, int64_t ldx, const void* w, const float* w_scale, const void* bias, void* y,
                    int64_t ldy, int64_t M, int64_t K, int64_t N) {
    if (M < 0 || K <= 0 || N <= 0) return fail(FP8LIN_ERR_SHAPE, "bad shape M=%lld K=%lld N=%lld", (long long)M, (long long)K, (long long)N);
    if (M > (1ll << 30) || K > (1ll << 30) || N > (1ll << 30)) return fail(FP8LIN_ERR_SHAPE, "dimension too large");
    if (K % 16 != 0) return fail(FP8LIN_ERR_SHAPE, "K=%lld must be a multiple of 16", (long long)K);
    if (M == 0) return FP8LIN_OK;
    if (!x || !w || !w_scale || !y) return fail(FP8LIN_ERR_NULL, "x, w_nk, w_scale and y must not be NULL");
    if (ldx < K || ldy < N) return fail(FP8LIN_ERR_SHAPE, "ldx=%lld < K or ldy=%lld < N", (long long)ldx, (long long)ldy);
    if (ldx % 8 != 0) return fail(FP8LIN_ERR_ALIGN, "ldx=%lld must be a multiple of 8 elements", (long long)ldx);
    if (!aligned16(x) || !aligned16(w) || !aligned16(w_scale) || (bias && !aligned16(bias)))
        return fail(FP8LIN_ERR_ALIGN, "x, w_nk, w_scale and bias must be 16-byte aligned");
    if (!check_arch()) return fail(FP8LIN_ERR_ARCH, "fp8lin kernels are built for sm_100a only");
    return FP8LIN_OK;
}

// Layers of up to ~17 MB with a short K (qkv, o_proj): up to 8 rows the mma.sync streaming kernel -- many small CTAs, its
// split-K slices handing their sums over inside a cluster -- starts and drains faster than the tcgen05 kernels.
bool small_layer(int64_t K, int64_t N) { return K <= 8192 && N <= 4736; }

bool w8a16_swap_eligible(int64_t M, int64_t K, int64_t N) {
    // measured (us, mma.sync kernel / tcgen05 kernel, which widens the weights on its way to TMEM): one row 3584 -> 37888
    // 23.1 / 21.0, 18944 -> 3584 15.7 / 14.0, 2048 -> 11008 8.1 / 6.9, but 3584 -> 4608 5.7 / 6.5, 3584 -> 3584 4.7 / 6.0,
    // 5120 -> 2560 5.4 / 6.2; 16 rows 26.9 / 22.8, 20.2 / 15.5, 10.1 / 7.8, 9.0 / 7.7, 7.8 / 6.9, 7.7 / 7.1
    const int min_m = g_tune.w8a16_swap_min_m >= 0 ? g_tune.w8a16_swap_min_m : (small_layer(K, N) ? 9 : 1);
    return g_tune.w8a16_swap_enable != 0 && M >= min_m && M <= 64;
}

// Routes by shape, kept per thread: the search for a plan takes 2 to 3 us of host time, as long as a small call's launch.  A
// fixed number of entries (a later shape replaces an earlier one); a knob that changes makes them all stale.
unsigned g_tune_version = 0;
template <class Route, class Make>
const Route& route_of(int64_t M, int64_t K, int64_t N, int flavour, Make make) {
    struct Entry {
        int64_t M = 0, K = 0, N = 0;
        int flavour = 0;
        unsigned version = 0;
        Route route;
    };
    static thread_local Entry table[128];
    const uint64_t h = ((uint64_t)M * 0x9e3779b97f4a7c15ull) ^ ((uint64_t)K * 0xc2b2ae3d27d4eb4full) ^ ((uint64_t)N * 0x165667b19e3779f9ull);
    Entry& e = table[((h >> 40) + (uint64_t)flavour) & 127];
    if (e.M != M || e.K != K || e.N != N || e.flavour != flavour || e.version != g_tune_version) {
        e.route = make();
        e.M = M; e.K = K; e.N = N; e.flavour = flavour; e.version = g_tune_version;
    }
    return e.route;
}

struct W8a16Route {
    bool pair = false;
    W8a16PairPlan plan{};
};
struct W8a8Route {
    bool pair = false;
    W8a8PairPlan plan{};
};

// W8A16 on CTA pairs with the weights widened into tensor memory and the caller's bf16 rows as the other operand.
// A knob that selects one of the other W8A16 routes switches it off.
bool w8a16_pair_wanted(int64_t M, int64_t K, int64_t N) {
    if (g_tune.w8a16_pair >= 0) return g_tune.w8a16_pair != 0;
    if (g_tune.w8a16_umma_min_m >= 0 || g_tune.w8a16_chunk_mb > 0 || g_tune.w8a16_swap_min_m >= 0 || g_tune.w8a16_swap_enable >= 0 ||
        g_tune.stream_splits > 0 || g_tune.swap_splits > 0)
        return false;
    if (M >= 65) return true;
    // 33 to 64 rows: pairs where the one-CTA kernel would not split K (it then widens every tile alone, 0.56 us per block at
    // 64 rows): 2048 -> 11008 11.0 us against 12.3, 2560 -> 9472 10.9 / 12.1, 3584 -> 37888 33.0 / 33.8; with slices it keeps
    // 3584 -> 4608 12.2 / 11.4, 18944 -> 3584 25.0 / 24.7
    if (M > 32 && plan_swap_w8a16(M, K, N, -1).splits == 1) return true;
    // from 49 rows also where the pairs do not split K and a third of them have a channel tile: 64 rows on 1280 -> 7168 6.2 / 8.2,
    // 2560 -> 9472 10.4 / 11.1; not 1280 -> 1536 (six tiles) 5.5 / 5.1
    return M > 48 && 3 * ((N + 255) / 256) >= sm_count() / 2 && plan_w8a16_pair(M, K, N, -1, -1).splits == 1;
}
// null: another kernel's
const W8a16PairPlan* w8a16_pair_route(int64_t M, int64_t K, int64_t N, int64_t ldy, const void* y) {
    if (N % 8 != 0 || ldy % 8 != 0 || !aligned16(y)) return nullptr;           // (the lanes store two channels at once; 8 and 16 bytes as in the other routes)
    const W8a16Route& r = route_of<W8a16Route>(M, K, N, 0, [&] {
        W8a16Route n;
        n.pair = w8a16_pair_wanted(M, K, N);
        if (n.pair) n.plan = plan_w8a16_pair(M, K, N, g_tune.w8a16_pair_tokens, g_tune.w8a16_pair_splits);
        return n;
    });
    return r.pair ? &r.plan : nullptr;
}

// Large-M W8A16: channel chunks of the weights are widened to f16 into scratch (small enough to stay
// in L2) and multiplied by the tcgen05 f16 GEMM; below this many rows the 64-row passes of the
// mma.sync kernel are cheaper than the per-chunk launches.
bool w8a16_umma_eligible(int64_t M, int64_t K, int64_t N, int64_t ldy, const void* y) {
    // measured on 3584 -> 37888: 128 rows 237 vs 132 us (passes win), 256 rows 270 vs 261 us (equal;
    // 32 vs 38 us on 3584 -> 4608), 1024 rows 319 vs 1032 us, 4096 rows 0.90 vs 4.1 ms
    const int min_m = g_tune.w8a16_umma_min_m >= 0 ? g_tune.w8a16_umma_min_m : 256;
    return min_m > 0 && M >= min_m && K % 8 == 0 && N % 8 == 0 && ldy % 8 == 0 && aligned16(y);
}

struct F16Chunks {
    int64_t chunk_tiles;     // 128-channel tile rows per chunk (even: a chunk is a multiple of 256 channels)
    int64_t n_chunks;
    size_t x16_bytes, w16_bytes;
};

F16Chunks plan_f16_chunks(int64_t M, int64_t K, int64_t N) {
    F16Chunks c;
    const int64_t ntiles = fp8lin::pack_ntiles(N);
    const size_t tile_row_bytes = (size_t)fp8lin::pack_kblocks(K) * 2 * fp8lin::kPackTileBytes;   // f16 bytes of 128 channels
    const size_t budget = (size_t)(g_tune.w8a16_chunk_mb > 0 ? g_tune.w8a16_chunk_mb : 64) << 20;
    // Chunks are counted in 256-channel column blocks (the GEMM's widest tile).  Every chunk is its own
    // GEMM launch of m_tiles x blocks tiles over 148 SMs, so the chunk size decides how many rounds of
    // tiles the whole call takes: try every size that fits the budget and keep the cheapest, a round
    // costing one tile's main loop and a chunk a fixed launch/ramp overhead.
    const int64_t nblocks = (ntiles + 1) / 2;
    int64_t max_blocks = (int64_t)(budget / (2 * tile_row_bytes));
    if (max_blocks < 1) max_blocks = 1;
    if (max_blocks > nblocks) max_blocks = nblocks;
    const int64_t m_tiles = (M + 127) / 128;
    const double t_tile = (double)fp8lin::pack_kblocks(K) * 2 * 0.115;     // us per 128x256 tile (64-element K blocks)
    auto rounds_of = [&](int64_t blocks) -> double {
        const int64_t tiles = m_tiles * blocks;
        if (tiles > (sm_count() / 2)) return (double)((tiles + (sm_count() - 1)) / sm_count());
        int64_t splits = sm_count() / tiles;                                       // few tiles: cluster split-K
        if (splits > 8) splits = 8;
        return 1.0 / (double)splits + 0.15;
    };
    double best_cost = 1e30;
    int64_t best_blocks = max_blocks;
    for (int64_t b = max_blocks; b >= 1 && b * 4 >= max_blocks; --b) {
        const int64_t full = nblocks / b, rest = nblocks - full * b;
        const double cost = (double)full * (rounds_of(b) * t_tile + 8.0) + (rest ? rounds_of(rest) * t_tile + 8.0 : 0.0);
        if (cost < best_cost - 1e-9) { best_cost = cost; best_blocks = b; }
    }
    const int64_t per = 2 * best_blocks;
    c.chunk_tiles = per;
    c.n_chunks = (ntiles + per - 1) / per;
    c.x16_bytes = align_up((size_t)M * K * 2, 256);
    c.w16_bytes = (size_t)per * tile_row_bytes;
    return c;
}

// CTA-pair GEMM (256 x 256 tiles over two SMs) instead of the one-CTA kernel: whichever finishes its rounds of tiles first.
// A K block of a round (74 pair tiles, or 148 tiles of 128 x 256 -- the same work) takes the pairs 0.44 us against 0.50:
// they stage and read a third fewer shared memory bytes per multiplication, and under the power limit that is clock; a call starts and ends 2.5 us later.  The
// pairs cannot cut a tile in two or split K, so the one-CTA kernel keeps short last rounds (half-width items, split-K tail)
// and few-tile shapes.  Fitted to eleven row counts from 128 to 16384 on six layer shapes: of 66 choices two are more than
// 4 % slower than the other kernel would have been, e.g. (us, pair / one CTA) 16384 x 3584 -> 3584 163 / 190, 16384 x 18944 -> 3584
// 868 / 920, 1031 x 18944 -> 3584 65 / 72, 4096 x 3584 -> 4608 54.6 / 61; but 4096 x 18944 -> 3584 248 / 235, 1536 x
// 18944 -> 3584 116 / 90, 256 x 3584 -> 4608 14.5 / 10.2.
bool pair_eligible(int64_t M, int64_t K, int64_t N) {
    if (g_tune.umma_pair >= 0) return g_tune.umma_pair != 0 && M > 64;
    const int sms = sm_count();
    const int64_t kblocks = (K + 127) / 128;
    const int64_t pair_tiles = ((M + 255) / 256) * ((N + 255) / 256);
    const int64_t pair_rounds = (pair_tiles + sms / 2 - 1) / (sms / 2);
    const UmmaPlan pl = plan_umma(M, K, N, g_tune.umma_bn, g_tune.umma_splits);
    if (pl.bn != 256) return false;
    const int64_t tiles = (int64_t)pl.m_tiles * pl.n_tiles;
    double rounds = (double)((tiles + sms - 1) / sms);
    if (pl.splits > 1) rounds = rounds / pl.splits + 0.12;
    else if (pl.tail_tiles) rounds += 1.0 / pl.tail_splits + 0.12 - 1.0;
    else if (pl.narrow_tiles) rounds += 0.52 - 1.0;
    return pair_rounds * kblocks * 0.44 + 6.0 < rounds * kblocks * 0.50 + 3.5;
}

// The same choice by how full the rounds are, without a model of their length: at least four rounds of pair tiles, the last
// one nearly full and no worse filled than the one-CTA kernel's.  Used where the result goes to several destinations (that
// epilogue has no split-K, so no tail to weigh), for the f16 operands of the scratch route, and in the variant name.
bool pair_rounds_full(int64_t M, int64_t N) {
    if (g_tune.umma_pair >= 0) return g_tune.umma_pair != 0 && M > 64;
    const int64_t nt = (N + 255) / 256;
    const int64_t pt = ((M + 255) / 256) * nt;
    const int64_t tiles = ((M + 127) / 128) * nt;
    if (pt < 4 * (sm_count() / 2)) return false;
    const double pair_fill = (double)pt / (double)(((pt + (sm_count() / 2 - 1)) / (sm_count() / 2)) * (sm_count() / 2));
    const double one_fill = (double)tiles / (double)(((tiles + (sm_count() - 1)) / sm_count()) * sm_count());
    return pair_fill >= 0.95 && pair_fill >= one_fill - 1e-9;
}

bool swap_eligible(int64_t M, int64_t K, int64_t N) {
    const int max_m = g_tune.stream_max_m >= 0 ? g_tune.stream_max_m : kDefaultStreamMaxM;
    // The tcgen05 kernel from the first row on, except on layers of up to ~17 MB with a short K (qkv, o_proj), where up to 8
    // rows the mma.sync streaming kernel starts and drains faster.  Measured, us, tcgen05 / streaming kernel, one row (eight
    // rows): 3584 -> 4608 6.1 / 5.8 (6.4 / 6.4), 3584 -> 3584 5.4 / 4.8 (5.7 / 5.4), 2048 -> 2048 3.8 / 3.7 (4.1 / 4.0); but 2048
    // -> 11008 6.9 / 9.1, 18944 -> 3584 13.7 / 16.6, 3584 -> 37888 20.6 / 23.7.  (5120 -> 2560 5.5 / 5.9 would now go the other
    // way; the line stays, because the two kernels add the products of an output in different orders: see plan_swap.)
    int min_m = g_tune.swap_min_m >= 0 ? g_tune.swap_min_m : 1;
    if (g_tune.swap_min_m < 0 && small_layer(K, N)) min_m = 9;
    return g_tune.swap_enable != 0 && M >= min_m && M <= 64 && M <= max_m;
}

// from this many rows on the swapped-operand kernel takes pre-quantised rows (one extra small
// pass, but nine ring slots instead of five or seven; measured faster from 17 rows up)
bool swap_prequant(int64_t M) {
    const int min_m = g_tune.swap_preq_min_m >= 0 ? g_tune.swap_preq_min_m : 17;
    return M >= min_m;
}

// Modelled microseconds of the kernels with 128- and 256-row tiles, to weigh them against plan_w8a8_pair's: rounds of tiles
// times K blocks, a cluster's hand-over or a last round cut in two where the plan has them; large calls of the CTA-pair GEMM
// are bound by power (0.385 us per pair tile and K block).  Fitted to the same row counts and shapes as that plan.
double umma_cost(const UmmaPlan& pl, int64_t K, int64_t N) {
    const double kblocks = (double)pack_kblocks(K), block = pl.bn == 256 ? 0.45 : (pl.bn == 128 ? 0.254 : 0.185);
    const int64_t tiles = (int64_t)pl.m_tiles * pl.n_tiles, sms = sm_count();
    if (pl.splits > 1) {
        const int64_t waves = (tiles + pl.slots - 1) / pl.slots;
        return (double)waves * (pl.kblocks_per_split * block + 1.17) + 1.81 * pl.bn / 128 + 3.14;
    }
    const double hbm = (double)K * (double)N / 5.5e6;                           // the weights, for few rows
    if (pl.narrow_tiles) return (double)(tiles / sms) * (kblocks * block + 0.49) + kblocks * block * 0.434 + 3.14;
    const double whole = (double)((tiles + sms - 1) / sms) * (kblocks * block + 0.49) + 3.14;
    return whole > hbm ? whole : hbm;
}
double umma_pair_cost(int64_t M, int64_t K, int64_t N) {
    const int64_t pairs = sm_count() / 2, tiles = ((M + 255) / 256) * ((N + 255) / 256);
    const double kblocks = (double)pack_kblocks(K), load = (double)(tiles < pairs ? tiles : pairs) / (double)pairs;
    const double chain = (double)((tiles + pairs - 1) / pairs) * (kblocks * 0.267 * (1.0 + 0.215 * load) + 0.06);
    const double power = (double)tiles * kblocks / (double)pairs * 0.385;
    return (chain > power ? chain : power) + 5.53;
}

// Knobs that select one of the other W8A8 routes.
bool other_w8a8_route_forced() {
    return g_tune.umma_pair >= 0 || g_tune.umma_bn > 0 || g_tune.umma_splits > 0 || g_tune.fuse_quant > 0 || g_tune.swap_min_m >= 0 ||
           g_tune.swap_enable >= 0 || g_tune.swap_splits > 0 || g_tune.swap_preq_min_m >= 0 || g_tune.stream_max_m >= 0 || g_tune.mlp_decode_fused > 0;
}

// W8A8 on CTA pairs with the rows as the MMA's N (umma_w8a8_pair.cu), K in as many slices as the sums of the other kernels
// have (see plan_swap); where the one-CTA GEMM would cut only its last tiles (its tail launch), the call stays there.
// Figures: us per call on rows that are codes, in a loop over weights from memory, this / the kernels it stands in for.
//   17 to 64 rows: where the one-CTA decode kernel does not split K (a pair's CTAs then stage half of the rows each: 64 rows
//     on 2048 -> 11008 6.2 / 7.8, 3584 -> 37888 23.1 / 24.2), and where the pairs are modelled faster (64 rows on 2048 -> 2048
//     4.84 / 4.96, 3584 -> 3584 6.92 / 7.07, 18944 -> 3584 14.7 / 15.3; not 8192 -> 1024 12.1 / 5.8).  Where K is split and bf16 rows bring a
//     quantiser in front, the decode kernel hides more of it (64 rows on 3584 -> 3584 8.6 / 7.9, 2048 -> 2048 6.4 / 6.3), which
//     this line does not weigh.
//   65 to 4096 rows: where modelled faster than both kernels with fixed tiles.  The model was fitted while the lanes stored the
//     results; since they leave by TMA a call of one K slice takes 0.86 of it.  (Several slices in one pair leave the same way and are weighed as they
//     were: up to 64 bf16 rows the decode kernel would lose its better cover of the quantiser by it, above that up to 10 % stays there, 128 rows
//     on 4096 -> 4096 9.3 / 10.2.)  Over eleven layer shapes (2048 -> 2048 .. 3584 ->
//     18944, 18944 -> 3584, 8192 -> 1024) and eighteen row counts from 17 on the choice is 0.2 % slower than the faster kernel, with the model as
//     it was 1.3 %: e.g. 700 rows on 3584 -> 4608 12.0 / 14.5, 1031 on 3584 -> 3584 13.0 / 14.2, 1500 on 11008 -> 2048 27.8 / 33.5, 256 on
//     3584 -> 18944 18.2 / 19.2, 512 on 2560 -> 9472 12.7 / 13.3, 4096 on 3584 -> 3584 40.3 / 45.1; not 160 on 8192 -> 1024 12.1 / 10.8.
//     Above 4096 rows the 256-row tiles are as good as full.
const W8a8PairPlan* w8a8_pair_route(int64_t M, int64_t K, int64_t N, int64_t ldy, const void* y) {
    if (N % 8 != 0 || ldy % 8 != 0 || !aligned16(y)) return nullptr;           // (whole sums leave by TMA, slices two channels per store)
    if (g_tune.w8a8_pair < 0 && (M < 17 || M > 4096 || other_w8a8_route_forced())) return nullptr;
    const W8a8Route& r = route_of<W8a8Route>(M, K, N, 0, [&] {
        W8a8Route n;
        if (g_tune.w8a8_pair == 0) return n;
        int slices = g_tune.w8a8_pair_slices;
        double other = 1e29;
        if (M <= 64) {
            const SwapPlan sp = plan_swap(M, K, N, -1, true);
            if (slices < 1) slices = sp.splits;
            other = sp.splits == 1 ? 1e29 : sp.cost;
        } else if (pair_rounds_full(M, N)) {
            if (slices < 1) slices = 1;
            other = umma_pair_cost(M, K, N);
        } else {
            const UmmaPlan pl = plan_umma(M, K, N, 0, 0);
            if (slices < 1) slices = pl.tail_tiles ? 0 : pl.splits;
            if (slices > 0) other = umma_cost(pl, K, N);
            if (pl.splits == 1 && other > umma_pair_cost(M, K, N)) other = umma_pair_cost(M, K, N);
        }
        n.plan = plan_w8a8_pair(M, K, N, false, slices, g_tune.w8a8_pair_tokens, g_tune.w8a8_pair_splits);
        n.pair = n.plan.cost * (n.plan.slices == 1 ? 0.86 : 1.0) < (g_tune.w8a8_pair > 0 ? 1e29 : other);
        return n;
    });
    return r.pair ? &r.plan : nullptr;
}
// The same kernel for gate_up of the fused MLP, with the activation in its epilogue.  Up to 64 rows the alternative is the
// decode kernel and a pass over its bf16 result, whose launch it saves: wherever that kernel would not split K.
const W8a8PairPlan* mlp_pair_route(int64_t M, int64_t H, int64_t I) {
    if (M < 17) return nullptr;
    if (g_tune.w8a8_pair < 0 && (M > 4096 || other_w8a8_route_forced())) return nullptr;
    const W8a8Route& r = route_of<W8a8Route>(M, H, 2 * I, 1, [&] {
        W8a8Route n;
        if (g_tune.w8a8_pair == 0) return n;
        const SwapPlan sp = M <= 64 ? plan_swap(M, H, 2 * I, -1, true) : SwapPlan{};
        n.plan = plan_w8a8_pair(M, H, 2 * I, true, M <= 64 ? sp.splits : 1, g_tune.w8a8_pair_tokens, 1);
        n.pair = n.plan.cost < (g_tune.w8a8_pair > 0 ? 1e30 : M <= 64 ? (sp.splits == 1 ? 1e29 : sp.cost + 2.0) : umma_pair_cost(M, H, 2 * I));
        return n;
    });
    return r.pair ? &r.plan : nullptr;
}

// Large-M W8A8 with the activation quantiser inside the GEMM: a short pass quantises the rows that the first
// round of tiles reads (tiles are walked in groups of eight tile rows), the kernel's quantiser warps do the
// rest while the tensor cores run.  Returns the number of rows for the pass; M = everything (no fusion).
int64_t prequant_rows(int64_t M, int64_t n_tiles, int tile_rows, int first_round_tiles) {
    // Off unless asked for.  Measured on a B200 (same process, alternating windows, 7B layer shapes at 4096 / 8192 /
    // 16384 rows): with the quantiser inside the GEMM qkv 77 / 141 / 274 us against 74 / 142 / 277 us with the
    // separate pass, o_proj 68 / 124 / 235 against 65 / 122 / 232, gate_up 511 / 1017 / 2045 against 513 / 1021 /
    // 2040, down 328 / 607 / 1180 against 296 / 579 / 1150.  These GEMMs run at the board's power limit (SM clock
    // 1.25-1.5 GHz of 1.965): hiding the pass does not remove its energy, the clock drops by what the extra warps
    // draw, and the pass alone runs at a power the GEMM never sees.
    if (g_tune.fuse_quant <= 0 || 3 + (M + 127) / 128 > kWsMaxCounters) return M;
    if (g_tune.fuse_quant > 1) {                      // forced split (tests): this many rows, rounded up to a row block
        const int64_t forced = ((int64_t)g_tune.fuse_quant + 127) / 128 * 128;
        return forced >= M ? M : forced;
    }
    const int64_t m_tiles = (M + tile_rows - 1) / tile_rows;
    const int64_t total = m_tiles * n_tiles;
    const int64_t first = total < first_round_tiles ? total : first_round_tiles;
    const int64_t groups = (first + 8 * n_tiles - 1) / (8 * n_tiles);
    const int64_t rows = groups * 8 * tile_rows;
    return rows >= M ? M : rows;
}

// Quantise rows [0, pre) in a pass of their own and hand the rest to the GEMM's quantiser warps.
// n_tiles, tile_rows, round_tiles: the GEMM's column tiles, rows per tile (128, or 256 on CTA pairs) and tiles in flight.
int start_quant(const void* x, int64_t ldx, const float* input_scale, unsigned char* xq, int64_t M, int64_t K, int64_t pre,
                const WsView& ws, UmmaArgs& a, cudaStream_t st, int64_t n_tiles, int tile_rows, int round_tiles) {
    cudaError_t e = launch_act_quant((const __nv_bfloat16*)x, ldx, input_scale, xq, pre, K, st);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "activation quantiser launch: %s", cudaGetErrorString(e));
    if (pre < M) {
        a.x = (const __nv_bfloat16*)x; a.ldx = (int)ldx; a.q_row_start = (int)pre; a.q_ctrl = ws.counters;
        // a CTA's next tile lies one round ahead: that many groups of eight tile rows, plus the group in progress
        // and one more so that the next blocks are ready when the tiles get there
        const int64_t groups_per_round = (round_tiles + 8 * n_tiles - 1) / (8 * n_tiles);
        a.q_lead = (int)((groups_per_round + 2) * 8 * (tile_rows / 128));
        if (g_tune.quant_lead >= 0) a.q_lead = g_tune.quant_lead;
    }
    return FP8LIN_OK;
}

bool umma_eligible(int64_t M, int64_t N, int64_t ldy, const void* y) {
    const int max_m = g_tune.stream_max_m >= 0 ? g_tune.stream_max_m : kDefaultStreamMaxM;
    return M > max_m && N % 8 == 0 && ldy % 8 == 0 && aligned16(y);
}

}  // namespace

namespace fp8lin {
static std::atomic<unsigned long long> g_launches{0};
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
bool device_is_sm100() { return check_arch() != 0; }
int sm_count() {
    static int cached = 0;
    if (cached > 0) return cached;
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0)
        return cached = n;
    cudaGetLastError();
    return 148;              // no device to ask (host-side planning only): not cached, a later call may have one
}
static int g_pdl = 1;
void set_pdl_enabled(int on) { g_pdl = on; }
int pdl_attribute(cudaLaunchAttribute* attr) {
    if (!g_pdl) return 0;
    attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr->val.programmaticStreamSerializationAllowed = 1;
    return 1;
}
int set_error(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}
}  // namespace fp8lin

extern "C" {

int fp8lin_version(void) { return FP8LIN_VERSION; }
unsigned long long fp8lin_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }
const char* fp8lin_last_error(void) { return g_err; }

size_t fp8lin_packed_bytes(int64_t K, int64_t N) {
    return (K > 0 && N > 0) ? (size_t)pack_ntiles(N) * (size_t)pack_kblocks(K) * kPackTileBytes : 0;
}

static int pack_common(const void* src, void* dst, int64_t K, int64_t N, bool src_is_kn, void* stream) {
    if (K <= 0 || N <= 0) return fail(FP8LIN_ERR_SHAPE, "bad shape K=%lld N=%lld", (long long)K, (long long)N);
    if (K % 16 != 0) return fail(FP8LIN_ERR_SHAPE, "K=%lld must be a multiple of 16", (long long)K);
    if (!src || !dst) return fail(FP8LIN_ERR_NULL, "source and destination must not be NULL");
    if (!aligned16(dst)) return fail(FP8LIN_ERR_ALIGN, "w_packed must be 16-byte aligned");
    cudaError_t e = launch_pack_tiles((const unsigned char*)src, (unsigned char*)dst, K, N, src_is_kn, (cudaStream_t)stream);
    if (e == cudaSuccess) e = launch_order((cudaStream_t)stream);       // (a linear behind this reads the weights before it waits)
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "prepack launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_prepack_weight(const void* qweight_kn, void* w_packed, int64_t K, int64_t N, void* stream) {
    return pack_common(qweight_kn, w_packed, K, N, true, stream);
}

int fp8lin_pack_weight_nk(const void* qweight_nk, void* w_packed, int64_t K, int64_t N, void* stream) {
    return pack_common(qweight_nk, w_packed, K, N, false, stream);
}

size_t fp8lin_workspace_bytes(int scheme, int64_t M, int64_t K, int64_t N) {
    if (M <= 0 || K <= 0 || N <= 0) return FP8LIN_WS_HEADER_BYTES;
    size_t body = 0;
    // streaming route (any M for W8A16; M <= 64 or odd shapes for W8A8)
    StreamPlan sp = plan_stream(scheme, M, K, N, g_tune.stream_splits);
    body = sp.partial_bytes;
    if (scheme == FP8LIN_W8A8_STATIC) {
        UmmaPlan up = plan_umma(M, K, N, g_tune.umma_bn, g_tune.umma_splits);
        size_t u = align_up((size_t)M * K, 256) + up.partial_bytes;
        if (u > body) body = u;
    } else if (w8a16_umma_eligible(M, K, N, 8, nullptr)) {
        F16Chunks c = plan_f16_chunks(M, K, N);
        if (c.x16_bytes + c.w16_bytes > body) body = c.x16_bytes + c.w16_bytes;
    }
    return FP8LIN_WS_HEADER_BYTES + align_up(body, 256);
}

static int run_stream(int scheme, const void* x, int64_t ldx, const void* w, const float* w_scale,
                      const float* input_scale, const void* bias, void* y, int64_t ldy, int64_t M, int64_t K,
                      int64_t N, void* workspace, size_t ws_bytes, cudaStream_t stream) {
    StreamPlan pl = plan_stream(scheme, M, K, N, g_tune.stream_splits);
    WsView ws = ws_view(workspace, ws_bytes);
    if (pl.splits > 1) {
        if (!workspace || ws.body_bytes < pl.partial_bytes)
            return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes", FP8LIN_WS_HEADER_BYTES + pl.partial_bytes);
    }
    StreamArgs a;
    a.x = (const __nv_bfloat16*)x; a.w = (const unsigned char*)w; a.w_scale = w_scale; a.input_scale = input_scale;
    a.bias = (const __nv_bfloat16*)bias; a.y = (__nv_bfloat16*)y;
    a.partial = workspace ? (float*)ws.body : nullptr; a.counters = workspace ? ws.counters : nullptr;
    a.status = workspace ? ws.status : nullptr;
    a.M = (int)M; a.K = (int)K; a.N = (int)N; a.ldx = (int)ldx; a.ldy = (int)ldy; a.k_per_split = pl.k_per_split;
    cudaError_t e = launch_stream(scheme, pl, a, stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "stream kernel launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_w8a16(const void* x, int64_t ldx, const void* w_nk, const float* w_scale, const void* bias, void* y,
                 int64_t ldy, int64_t M, int64_t K, int64_t N, void* workspace, size_t workspace_bytes,
                 void* stream) {
    int rc = validate_common(x, ldx, w_nk, w_scale, bias, y, ldy, M, K, N);
    if (rc != FP8LIN_OK || M == 0) return rc;
    const W8a16PairPlan* pair = workspace && workspace_bytes >= FP8LIN_WS_HEADER_BYTES ? w8a16_pair_route(M, K, N, ldy, y) : nullptr;
    if (pair) {
        UmmaArgs a;
        a.xq = nullptr; a.w = (const unsigned char*)w_nk; a.w_scale = w_scale; a.input_scale = nullptr;
        a.bias = (const __nv_bfloat16*)bias; a.y = (__nv_bfloat16*)y; a.partial = nullptr; a.counters = nullptr;
        a.status = ws_view(workspace, workspace_bytes).status; a.M = (int)M; a.K = (int)K; a.N = (int)N; a.ldy = (int)ldy;
        const char* why = nullptr;
        cudaError_t e = launch_w8a16_pair(*pair, a, x, ldx, (cudaStream_t)stream, &why);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "tcgen05 W8A16 pair kernel launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
        return FP8LIN_OK;
    }
    if (w8a16_swap_eligible(M, K, N) && workspace) {
        SwapPlan sp = plan_swap_w8a16(M, K, N, g_tune.swap_splits);
        UmmaArgs a;
        a.xq = nullptr; a.w = (const unsigned char*)w_nk; a.w_scale = w_scale; a.input_scale = nullptr;
        a.bias = (const __nv_bfloat16*)bias; a.y = (__nv_bfloat16*)y; a.partial = nullptr; a.counters = nullptr;
        a.status = ws_view(workspace, workspace_bytes).status; a.M = (int)M; a.K = (int)K; a.N = (int)N; a.ldy = (int)ldy;
        const char* why = nullptr;
        cudaError_t e = launch_swap_w8a16(sp, a, x, ldx, (cudaStream_t)stream, &why);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "tcgen05 W8A16 decode kernel launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
        return FP8LIN_OK;
    }
    if (w8a16_umma_eligible(M, K, N, ldy, y)) {
        cudaStream_t st = (cudaStream_t)stream;
        const F16Chunks c = plan_f16_chunks(M, K, N);
        WsView ws = ws_view(workspace, workspace_bytes);
        if (!workspace || ws.body_bytes < c.x16_bytes + c.w16_bytes)
            return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes",
                        (size_t)FP8LIN_WS_HEADER_BYTES + c.x16_bytes + c.w16_bytes);
        unsigned char* x16 = ws.body;
        unsigned char* w16 = ws.body + c.x16_bytes;
        cudaError_t e = launch_x_to_f16((const __nv_bfloat16*)x, ldx, x16, M, K, st);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "f16 activation pass launch: %s", cudaGetErrorString(e));
        const int64_t kb = pack_kblocks(K);
        for (int64_t ci = 0; ci < c.n_chunks; ++ci) {
            const int64_t t0 = ci * c.chunk_tiles;
            const int64_t n0 = t0 * kPackTile;
            const int64_t nc = (N - n0) < c.chunk_tiles * kPackTile ? (N - n0) : c.chunk_tiles * kPackTile;
            const int64_t tiles = pack_ntiles(nc);
            e = launch_dequant_tiles_f16((const unsigned char*)w_nk + (size_t)t0 * kb * kPackTileBytes, w16,
                                         tiles * kb * kPackTileBytes, st);
            if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "f16 weight pass launch: %s", cudaGetErrorString(e));
            UmmaPlan pl = plan_umma(M, 2 * kb * kPackTile, nc, g_tune.umma_bn, g_tune.umma_splits);
            UmmaArgs a;
            a.xq = x16; a.w = w16; a.w_scale = w_scale + n0; a.input_scale = nullptr;
            a.bias = bias ? (const __nv_bfloat16*)bias + n0 : nullptr; a.y = (__nv_bfloat16*)y + n0;
            a.partial = nullptr; a.counters = ws.counters; a.status = ws.status;
            a.M = (int)M; a.K = (int)K; a.N = (int)nc; a.ldy = (int)ldy;
            const char* why = nullptr;
            e = pair_rounds_full(M, nc) ? launch_umma_pair(true, a, st, &why) : launch_umma_f16(pl, a, st, &why);
            if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "tcgen05 f16 GEMM launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
        }
        return FP8LIN_OK;
    }
    return run_stream(FP8LIN_W8A16, x, ldx, w_nk, w_scale, nullptr, bias, y, ldy, M, K, N, workspace,
                      workspace_bytes, (cudaStream_t)stream);
}

namespace {

// W8A8 linear whose activations are already e4m3 (row pitch K).
int run_w8a8_prequantised(const unsigned char* xq, const void* w, const float* w_scale, const float* input_scale,
                          const void* bias, void* y, int64_t ldy, int64_t M, int64_t K, int64_t N, const WsView& ws,
                          cudaStream_t st) {
    UmmaArgs a;
    a.xq = xq; a.w = (const unsigned char*)w; a.w_scale = w_scale; a.input_scale = input_scale;
    a.bias = (const __nv_bfloat16*)bias; a.y = (__nv_bfloat16*)y; a.partial = nullptr; a.counters = ws.counters;
    a.status = ws.status; a.M = (int)M; a.K = (int)K; a.N = (int)N; a.ldy = (int)ldy;
    const char* why = nullptr;
    cudaError_t e;
    if (const W8a8PairPlan* pair = w8a8_pair_route(M, K, N, ldy, y)) {
        e = launch_w8a8_pair(*pair, a, st, &why);
    } else if (M <= 64) {
        SwapPlan sp = plan_swap(M, K, N, g_tune.swap_splits, true);
        e = launch_swap_w8a8(sp, a, nullptr, 0, st, &why);
    } else if (pair_eligible(M, K, N)) {
        e = launch_umma_pair(false, a, st, &why);
    } else {
        UmmaPlan pl = plan_umma(M, K, N, g_tune.umma_bn, g_tune.umma_splits);
        e = launch_umma_w8a8(pl, a, st, &why);
    }
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "W8A8 linear launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
    return FP8LIN_OK;
}

}  // namespace

int fp8lin_w8a8(const void* x, int64_t ldx, const void* w_nk, const float* w_scale, const float* input_scale,
                const void* bias, void* y, int64_t ldy, int64_t M, int64_t K, int64_t N, void* workspace,
                size_t workspace_bytes, void* stream) {
    int rc = validate_common(x, ldx, w_nk, w_scale, bias, y, ldy, M, K, N);
    if (rc != FP8LIN_OK || M == 0) return rc;
    if (!input_scale) return fail(FP8LIN_ERR_NULL, "input_scale must not be NULL");
    cudaStream_t st = (cudaStream_t)stream;
    if (w8a8_pair_route(M, K, N, ldy, y)) {
        WsView wsv = ws_view(workspace, workspace_bytes);
        if (!workspace || wsv.body_bytes < align_up((size_t)M * K, 256))
            return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes", FP8LIN_WS_HEADER_BYTES + align_up((size_t)M * K, 256));
        cudaError_t qe = launch_act_quant((const __nv_bfloat16*)x, ldx, input_scale, wsv.body, M, K, st);
        if (qe != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "activation quantiser launch: %s", cudaGetErrorString(qe));
        return run_w8a8_prequantised(wsv.body, w_nk, w_scale, input_scale, bias, y, ldy, M, K, N, wsv, st);
    }
    if (swap_eligible(M, K, N)) {
        const bool preq = swap_prequant(M);
        SwapPlan sp = plan_swap(M, K, N, g_tune.swap_splits, preq);
        WsView wsv = ws_view(workspace, workspace_bytes);
        if (!workspace) return fail(FP8LIN_ERR_WORKSPACE, "workspace (at least the %d-byte header) is required", FP8LIN_WS_HEADER_BYTES);
        UmmaArgs a;
        a.xq = nullptr;
        if (preq) {
            if (wsv.body_bytes < align_up((size_t)M * K, 256))
                return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes", FP8LIN_WS_HEADER_BYTES + align_up((size_t)M * K, 256));
            cudaError_t qe = launch_act_quant((const __nv_bfloat16*)x, ldx, input_scale, wsv.body, M, K, st);
            if (qe != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "activation quantiser launch: %s", cudaGetErrorString(qe));
            a.xq = wsv.body;
        } a.w = (const unsigned char*)w_nk; a.w_scale = w_scale; a.input_scale = input_scale;
        a.bias = (const __nv_bfloat16*)bias; a.y = (__nv_bfloat16*)y; a.partial = nullptr; a.counters = nullptr;
        a.status = wsv.status; a.M = (int)M; a.K = (int)K; a.N = (int)N; a.ldy = (int)ldy;
        const char* why = nullptr;
        cudaError_t e = launch_swap_w8a8(sp, a, x, ldx, st, &why);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "tcgen05 decode kernel launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
        return FP8LIN_OK;
    }
    if (!umma_eligible(M, N, ldy, y))
        return run_stream(FP8LIN_W8A8_STATIC, x, ldx, w_nk, w_scale, input_scale, bias, y, ldy, M, K, N, workspace,
                          workspace_bytes, st);

    UmmaPlan pl = plan_umma(M, K, N, g_tune.umma_bn, g_tune.umma_splits);
    WsView ws = ws_view(workspace, workspace_bytes);
    const size_t xq_bytes = align_up((size_t)M * K, 256);
    if (!workspace || ws.body_bytes < xq_bytes + pl.partial_bytes)
        return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes",
                    FP8LIN_WS_HEADER_BYTES + xq_bytes + pl.partial_bytes);
    unsigned char* xq = ws.body;
    UmmaArgs a;
    a.xq = xq; a.w = (const unsigned char*)w_nk; a.w_scale = w_scale; a.input_scale = input_scale;
    a.bias = (const __nv_bfloat16*)bias; a.y = (__nv_bfloat16*)y;
    a.partial = (float*)(ws.body + xq_bytes); a.counters = ws.counters; a.status = ws.status;
    a.M = (int)M; a.K = (int)K; a.N = (int)N; a.ldy = (int)ldy;
    const bool pair = pair_eligible(M, K, N);
    const int64_t pre = pair ? prequant_rows(M, (N + 255) / 256, 256, sm_count() / 2)
                             : (pl.splits > 1 ? M : prequant_rows(M, pl.n_tiles, 128, sm_count()));
    rc = pair ? start_quant(x, ldx, input_scale, xq, M, K, pre, ws, a, st, (N + 255) / 256, 256, sm_count() / 2)
              : start_quant(x, ldx, input_scale, xq, M, K, pre, ws, a, st, pl.n_tiles, 128, sm_count());
    if (rc != FP8LIN_OK) return rc;
    const char* why = nullptr;
    cudaError_t e = pair ? launch_umma_pair(false, a, st, &why) : launch_umma_w8a8(pl, a, st, &why);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "tcgen05 GEMM launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
    return FP8LIN_OK;
}

static int w8a8_to_destinations(const void* x, int64_t ldx, const void* w_nk, const float* w_scale, const float* input_scale,
                                const void* bias, int n_dst, void* const* dst_ptrs, int64_t ld_dst, int64_t band_rows, int64_t M,
                                int64_t K, int64_t N, void* workspace, size_t workspace_bytes, void* stream) {
    if (n_dst < 1 || n_dst > 8 || !dst_ptrs) return fail(FP8LIN_ERR_ARG, "n_dst must be 1..8 and dst_ptrs non-NULL");
    for (int d = 0; d < n_dst; ++d)
        if (!dst_ptrs[d] || !aligned16(dst_ptrs[d])) return fail(FP8LIN_ERR_ALIGN, "destination %d is NULL or not 16-byte aligned", d);
    int rc = validate_common(x, ldx, w_nk, w_scale, bias, dst_ptrs[0], ld_dst, M, K, N);
    if (rc != FP8LIN_OK || M == 0) return rc;
    if (!input_scale) return fail(FP8LIN_ERR_NULL, "input_scale must not be NULL");
    if (N % 8 != 0 || ld_dst % 8 != 0) return fail(FP8LIN_ERR_SHAPE, "N and ld_dst must be multiples of 8");
    if (band_rows != 0 && (band_rows < 32 || band_rows % 32 != 0 || band_rows * n_dst < M))
        return fail(FP8LIN_ERR_SHAPE, "band_rows=%lld must be a multiple of 32 with band_rows * n_dst >= M", (long long)band_rows);
    cudaStream_t st = (cudaStream_t)stream;
    UmmaPlan pl = plan_umma(M, K, N, g_tune.umma_bn, 1);      // the multi-destination epilogue exists in the non-split kernels only
    pl.tail_tiles = 0;
    WsView ws = ws_view(workspace, workspace_bytes);
    const size_t xq_bytes = align_up((size_t)M * K, 256);
    if (!workspace || ws.body_bytes < xq_bytes)
        return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes", FP8LIN_WS_HEADER_BYTES + xq_bytes);
    UmmaArgs a;
    a.xq = ws.body; a.w = (const unsigned char*)w_nk; a.w_scale = w_scale; a.input_scale = input_scale;
    a.bias = (const __nv_bfloat16*)bias; a.y = (__nv_bfloat16*)dst_ptrs[0]; a.partial = nullptr; a.counters = ws.counters;
    a.status = ws.status; a.M = (int)M; a.K = (int)K; a.N = (int)N; a.ldy = (int)ld_dst;
    const bool pair = pair_rounds_full(M, N);
    rc = pair ? start_quant(x, ldx, input_scale, ws.body, M, K, prequant_rows(M, (N + 255) / 256, 256, sm_count() / 2), ws, a, st,
                            (N + 255) / 256, 256, sm_count() / 2)
              : start_quant(x, ldx, input_scale, ws.body, M, K, prequant_rows(M, pl.n_tiles, 128, sm_count()), ws, a, st, pl.n_tiles, 128,
                            sm_count());
    if (rc != FP8LIN_OK) return rc;
    const char* why = nullptr;
    cudaError_t e = pair ? launch_umma_pair(false, a, st, &why, n_dst, dst_ptrs, ld_dst, band_rows)
                         : launch_umma_w8a8(pl, a, st, &why, n_dst, dst_ptrs, ld_dst, band_rows);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "tcgen05 GEMM launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
    return FP8LIN_OK;
}

int fp8lin_w8a8_scatter(const void* x, int64_t ldx, const void* w_nk, const float* w_scale, const float* input_scale,
                        const void* bias, int n_dst, void* const* dst_ptrs, int64_t ld_dst, int64_t M, int64_t K, int64_t N,
                        void* workspace, size_t workspace_bytes, void* stream) {
    return w8a8_to_destinations(x, ldx, w_nk, w_scale, input_scale, bias, n_dst, dst_ptrs, ld_dst, 0, M, K, N, workspace,
                                workspace_bytes, stream);
}

int fp8lin_w8a8_reduce_scatter(const void* x, int64_t ldx, const void* w_nk, const float* w_scale, const float* input_scale,
                               const void* bias, int n_dst, void* const* dst_ptrs, int64_t ld_dst, int64_t band_rows, int64_t M,
                               int64_t K, int64_t N, void* workspace, size_t workspace_bytes, void* stream) {
    if (band_rows <= 0) return fail(FP8LIN_ERR_SHAPE, "band_rows must be positive");
    return w8a8_to_destinations(x, ldx, w_nk, w_scale, input_scale, bias, n_dst, dst_ptrs, ld_dst, band_rows, M, K, N, workspace,
                                workspace_bytes, stream);
}

// ---- fused MLP: y = down( silu(gate(x)) * up(x) ), both projections W8A8-static -----------------------
namespace {

struct MlpLayout {
    size_t inner;       // scratch of the gate_up linear itself (quantised x, split-K partials)
    size_t gu_off, hq_off, total;
};

MlpLayout mlp_layout(int64_t M, int64_t H, int64_t I) {
    MlpLayout l;
    size_t inner = fp8lin_workspace_bytes(FP8LIN_W8A8_STATIC, M, H, 2 * I) - FP8LIN_WS_HEADER_BYTES;
    const size_t xq = align_up((size_t)M * H, 256);
    if (xq > inner) inner = xq;
    l.inner = align_up(inner, 256);
    l.gu_off = l.inner;
    const size_t gu = M <= kDefaultStreamMaxM ? align_up((size_t)M * 2 * I * 2, 256) : 0;   // bf16 gate_up result, small batches only
    l.hq_off = l.gu_off + gu;
    l.total = l.hq_off + align_up((size_t)M * I, 256);
    return l;
}

}  // namespace

size_t fp8lin_mlp_workspace_bytes(int64_t M, int64_t H, int64_t I, int64_t N) {
    (void)N;
    if (M <= 0 || H <= 0 || I <= 0) return FP8LIN_WS_HEADER_BYTES;
    return FP8LIN_WS_HEADER_BYTES + mlp_layout(M, H, I).total;
}

static int mlp_w8a8_impl(const void* x, int64_t ldx, bool x_is_e4m3, const void* w_gate_up, const float* gate_up_scale,
                         const float* gate_up_input_scale, const void* gate_up_bias, const void* w_down,
                         const float* down_scale, const float* down_input_scale, const void* down_bias, void* y, int64_t ldy,
                         int64_t M, int64_t H, int64_t I, int64_t N, void* workspace, size_t workspace_bytes, void* stream) {
    if (I <= 0 || I % 128 != 0) return fail(FP8LIN_ERR_SHAPE, "the intermediate size must be a positive multiple of 128 (got %lld)", (long long)I);
    int rc = validate_common(x, ldx, w_gate_up, gate_up_scale, gate_up_bias, y, 2 * I, M, H, 2 * I);   // (its output is internal)
    if (rc != FP8LIN_OK) return rc;
    rc = validate_common(x, I, w_down, down_scale, down_bias, y, ldy, M, I, N);      // (the down input is internal, pitch I)
    if (rc != FP8LIN_OK || M == 0) return rc;
    if (!gate_up_input_scale || !down_input_scale) return fail(FP8LIN_ERR_NULL, "both input scales are required");
    if (N % 8 != 0 || ldy % 8 != 0) return fail(FP8LIN_ERR_SHAPE, "N and ldy must be multiples of 8");
    const MlpLayout l = mlp_layout(M, H, I);
    WsView ws = ws_view(workspace, workspace_bytes);
    if (!workspace || ws.body_bytes < l.total)
        return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes", (size_t)FP8LIN_WS_HEADER_BYTES + l.total);
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char* hq = ws.body + l.hq_off;
    if (x_is_e4m3 && M <= 16 && g_tune.mlp_decode_fused > 0) {
        // Opt-in: up to 16 pre-quantised rows, clusters of two CTAs of the decode kernel take (gate, up) tile pairs, the
        // up CTA hands its values to the gate CTA, which writes e4m3 h itself (one launch fewer, no bf16 gate_up round
        // trip, same bits).  Off by default, it buys nothing: 55.9 us per 7B decoder layer at one row against 55.5 us
        // with the separate 3 us activation pass (58.7 against 58.3 at 16 rows; 28 layers under one CUDA graph) -- the
        // hand-over buffer costs the ring its sixth slot and the hand-over sits on the kernel's tail.  A first form
        // (both tiles in one CTA with a 12-slot ring, one CTA per SM) was slower still: 58.6 us.
        UmmaArgs a;
        a.xq = (const unsigned char*)x; a.w = (const unsigned char*)w_gate_up; a.w_scale = gate_up_scale; a.input_scale = gate_up_input_scale;
        a.bias = (const __nv_bfloat16*)gate_up_bias; a.y = nullptr; a.partial = nullptr; a.counters = nullptr;
        a.status = ws.status; a.M = (int)M; a.K = (int)H; a.N = (int)(2 * I); a.ldy = 0;
        a.hq = hq; a.h_scale = down_input_scale;
        const char* why = nullptr;
        cudaError_t e = launch_swap_gate_up(a, st, &why);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "decode gate_up launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
    } else if (const W8a8PairPlan* pair = mlp_pair_route(M, H, I)) {
        UmmaArgs a;
        a.xq = x_is_e4m3 ? (const unsigned char*)x : ws.body; a.w = (const unsigned char*)w_gate_up; a.w_scale = gate_up_scale;
        a.input_scale = gate_up_input_scale; a.bias = (const __nv_bfloat16*)gate_up_bias; a.y = nullptr; a.partial = nullptr;
        a.counters = nullptr; a.status = ws.status; a.M = (int)M; a.K = (int)H; a.N = (int)(2 * I); a.ldy = 0;
        a.hq = hq; a.h_scale = down_input_scale;
        if (!x_is_e4m3) {
            cudaError_t qe = launch_act_quant((const __nv_bfloat16*)x, ldx, gate_up_input_scale, ws.body, M, H, st);
            if (qe != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "activation quantiser launch: %s", cudaGetErrorString(qe));
        }
        const char* why = nullptr;
        cudaError_t e = launch_w8a8_pair(*pair, a, st, &why);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "fused gate_up launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
    } else if (M <= kDefaultStreamMaxM) {
        // small batches: gate_up through the decode kernels into a bf16 buffer, one pass for silu * up + quantise
        __nv_bfloat16* gu = (__nv_bfloat16*)(ws.body + l.gu_off);
        if (x_is_e4m3) {
            WsView inner = ws_view(workspace, FP8LIN_WS_HEADER_BYTES + l.inner);
            rc = run_w8a8_prequantised((const unsigned char*)x, w_gate_up, gate_up_scale, gate_up_input_scale, gate_up_bias, gu, 2 * I,
                                       M, H, 2 * I, inner, st);
        } else {
            rc = fp8lin_w8a8(x, ldx, w_gate_up, gate_up_scale, gate_up_input_scale, gate_up_bias, gu, 2 * I, M, H, 2 * I, workspace,
                             FP8LIN_WS_HEADER_BYTES + l.inner, stream);
        }
        if (rc != FP8LIN_OK) return rc;
        cudaError_t e = launch_silu_mul_quant_interleaved(gu, down_input_scale, hq, M, I, st);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "silu-multiply pass launch: %s", cudaGetErrorString(e));
    } else {
        unsigned char* xq = x_is_e4m3 ? (unsigned char*)const_cast<void*>(x) : ws.body;
        UmmaArgs a;
        a.xq = xq; a.w = (const unsigned char*)w_gate_up; a.w_scale = gate_up_scale; a.input_scale = gate_up_input_scale;
        a.bias = (const __nv_bfloat16*)gate_up_bias; a.y = nullptr; a.partial = nullptr; a.counters = ws.counters;
        a.status = ws.status; a.M = (int)M; a.K = (int)H; a.N = (int)(2 * I); a.ldy = 0;
        if (!x_is_e4m3) {
            rc = start_quant(x, ldx, gate_up_input_scale, xq, M, H, prequant_rows(M, (2 * I + 255) / 256, 256, sm_count() / 2), ws, a, st,
                             (2 * I + 255) / 256, 256, sm_count() / 2);
            if (rc != FP8LIN_OK) return rc;
        }
        const char* why = nullptr;
        cudaError_t e = launch_umma_pair_mlp(a, hq, down_input_scale, st, &why);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "fused gate_up launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
    }
    return run_w8a8_prequantised(hq, w_down, down_scale, down_input_scale, down_bias, y, ldy, M, I, N, ws, st);
}

int fp8lin_w8a8_preq(const void* xq, const void* w_nk, const float* w_scale, const float* input_scale, const void* bias,
                     void* y, int64_t ldy, int64_t M, int64_t K, int64_t N, void* workspace, size_t workspace_bytes,
                     void* stream) {
    int rc = validate_common(xq, K, w_nk, w_scale, bias, y, ldy, M, K, N);      // (xq rows are K bytes apart)
    if (rc != FP8LIN_OK || M == 0) return rc;
    if (!input_scale) return fail(FP8LIN_ERR_NULL, "input_scale must not be NULL");
    if (N % 8 != 0 || ldy % 8 != 0 || !aligned16(y)) return fail(FP8LIN_ERR_ALIGN, "N and ldy must be multiples of 8 and y 16-byte aligned");
    if (!workspace || workspace_bytes < FP8LIN_WS_HEADER_BYTES)
        return fail(FP8LIN_ERR_WORKSPACE, "workspace (at least the %d-byte header) is required", FP8LIN_WS_HEADER_BYTES);
    return run_w8a8_prequantised((const unsigned char*)xq, w_nk, w_scale, input_scale, bias, y, ldy, M, K, N,
                                 ws_view(workspace, workspace_bytes), (cudaStream_t)stream);
}

int fp8lin_rmsnorm_quant(const void* x, int64_t ldx, void* residual, int64_t ld_res, const void* weight, float eps,
                         const float* input_scale, void* xq, void* y, int64_t ldy, int64_t M, int64_t H, void* stream) {
    if (M < 0 || H <= 0 || H % 8 != 0 || H > 8192)
        return fail(FP8LIN_ERR_SHAPE, "bad shape M=%lld H=%lld (H a multiple of 8, at most 8192)", (long long)M, (long long)H);
    if (M == 0) return FP8LIN_OK;
    if (!x || !weight || (!xq && !y)) return fail(FP8LIN_ERR_NULL, "x, weight and at least one of xq / y must not be NULL");
    if (xq && !input_scale) return fail(FP8LIN_ERR_NULL, "input_scale is required when xq is asked for");
    if (ldx < H || (residual && ld_res < H) || (y && ldy < H)) return fail(FP8LIN_ERR_SHAPE, "a row stride is smaller than H");
    if (ldx % 8 != 0 || (residual && ld_res % 8 != 0) || (y && ldy % 8 != 0))
        return fail(FP8LIN_ERR_ALIGN, "row strides must be multiples of 8 elements");
    if (!aligned16(x) || !aligned16(weight) || (residual && !aligned16(residual)) || (y && !aligned16(y)) ||
        (xq && (reinterpret_cast<uintptr_t>(xq) & 7) != 0))
        return fail(FP8LIN_ERR_ALIGN, "x, residual, weight and y must be 16-byte aligned, xq 8-byte aligned");
    if (!(eps >= 0.f)) return fail(FP8LIN_ERR_ARG, "eps must not be negative");
    if (!check_arch()) return fail(FP8LIN_ERR_ARCH, "fp8lin kernels are built for sm_100a only");
    cudaError_t e = launch_rmsnorm_quant((const __nv_bfloat16*)x, ldx, (__nv_bfloat16*)residual, ld_res, (const __nv_bfloat16*)weight,
                                         eps, input_scale, (unsigned char*)xq, (__nv_bfloat16*)y, ldy, M, H, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "RMSNorm launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_mlp_w8a8(const void* x, int64_t ldx, const void* w_gate_up, const float* gate_up_scale,
                    const float* gate_up_input_scale, const void* gate_up_bias, const void* w_down,
                    const float* down_scale, const float* down_input_scale, const void* down_bias, void* y, int64_t ldy,
                    int64_t M, int64_t H, int64_t I, int64_t N, void* workspace, size_t workspace_bytes, void* stream) {
    return mlp_w8a8_impl(x, ldx, false, w_gate_up, gate_up_scale, gate_up_input_scale, gate_up_bias, w_down, down_scale,
                         down_input_scale, down_bias, y, ldy, M, H, I, N, workspace, workspace_bytes, stream);
}

int fp8lin_mlp_w8a8_preq(const void* xq, const void* w_gate_up, const float* gate_up_scale,
                         const float* gate_up_input_scale, const void* gate_up_bias, const void* w_down,
                         const float* down_scale, const float* down_input_scale, const void* down_bias, void* y, int64_t ldy,
                         int64_t M, int64_t H, int64_t I, int64_t N, void* workspace, size_t workspace_bytes, void* stream) {
    return mlp_w8a8_impl(xq, (H + 7) / 8 * 8, true, w_gate_up, gate_up_scale, gate_up_input_scale, gate_up_bias, w_down, down_scale,
                         down_input_scale, down_bias, y, ldy, M, H, I, N, workspace, workspace_bytes, stream);
}

int fp8lin_sum_slots(const void* slots, int n_slots, int64_t slot_stride, int64_t ld_slot, void* y, int64_t ldy,
                     int64_t M, int64_t N, void* stream) {
    if (n_slots < 1 || M < 0 || N <= 0 || N % 8 != 0 || ld_slot % 8 != 0 || ldy % 8 != 0 || slot_stride % 8 != 0)
        return fail(FP8LIN_ERR_SHAPE, "bad shape: N, ld_slot, ldy and slot_stride must be multiples of 8");
    if (M == 0) return FP8LIN_OK;
    if (!slots || !y) return fail(FP8LIN_ERR_NULL, "slots and y must not be NULL");
    if (!aligned16(slots) || !aligned16(y)) return fail(FP8LIN_ERR_ALIGN, "slots and y must be 16-byte aligned");
    cudaError_t e = launch_sum_slots((const __nv_bfloat16*)slots, n_slots, slot_stride, (__nv_bfloat16*)y, ldy, M, N, ld_slot,
                                     (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "slot sum launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_sum_slots_gather(const void* slots, int n_slots, int64_t slot_stride, int64_t ld_slot, int n_dst, void* const* dst_ptrs,
                            int64_t ld_dst, int64_t dst_row, int64_t M, int64_t N, void* stream) {
    if (n_slots < 1 || M < 0 || N <= 0 || N % 8 != 0 || ld_slot % 8 != 0 || ld_dst % 8 != 0 || slot_stride % 8 != 0 || dst_row < 0)
        return fail(FP8LIN_ERR_SHAPE, "bad shape: N, ld_slot, ld_dst and slot_stride must be multiples of 8");
    if (n_dst < 1 || n_dst > 8 || !dst_ptrs) return fail(FP8LIN_ERR_ARG, "n_dst must be 1..8 and dst_ptrs non-NULL");
    if (M == 0) return FP8LIN_OK;
    if (!slots || !aligned16(slots)) return fail(FP8LIN_ERR_ALIGN, "slots must be non-NULL and 16-byte aligned");
    SumDst dst;
    dst.n = n_dst;
    for (int d = 0; d < n_dst; ++d) {
        if (!dst_ptrs[d] || !aligned16(dst_ptrs[d])) return fail(FP8LIN_ERR_ALIGN, "destination %d is NULL or not 16-byte aligned", d);
        dst.y[d] = (__nv_bfloat16*)dst_ptrs[d] + dst_row * ld_dst;
    }
    cudaError_t e = launch_sum_slots_gather((const __nv_bfloat16*)slots, n_slots, slot_stride, ld_slot, dst, ld_dst, M, N,
                                            (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "slot sum launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_quantize_weight(const void* w, int w_is_f32, int64_t ldw, void* qweight_nk, float* weight_scale, int64_t N,
                           int64_t K, void* stream) {
    if (N < 0 || K <= 0 || K % 2 != 0 || ldw < K) return fail(FP8LIN_ERR_SHAPE, "bad shape N=%lld K=%lld ldw=%lld (K must be even)", (long long)N, (long long)K, (long long)ldw);
    if (N == 0) return FP8LIN_OK;
    if (!w || !qweight_nk || !weight_scale) return fail(FP8LIN_ERR_NULL, "w, qweight_nk and weight_scale must not be NULL");
    if ((reinterpret_cast<uintptr_t>(qweight_nk) & 1) != 0) return fail(FP8LIN_ERR_ALIGN, "qweight_nk must be 2-byte aligned");
    if (!check_arch()) return fail(FP8LIN_ERR_ARCH, "fp8lin kernels are built for sm_100a only");
    cudaError_t e = launch_quantize_weight(w, w_is_f32 != 0, ldw, (unsigned char*)qweight_nk, weight_scale, N, K, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "weight quantiser launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_abs_max(const void* x, int64_t ldx, int64_t M, int64_t K, float* amax, void* stream) {
    if (M < 0 || K <= 0 || K % 8 != 0 || ldx < K || ldx % 8 != 0) return fail(FP8LIN_ERR_SHAPE, "bad shape M=%lld K=%lld ldx=%lld (multiples of 8)", (long long)M, (long long)K, (long long)ldx);
    if (M == 0) return FP8LIN_OK;
    if (!x || !amax) return fail(FP8LIN_ERR_NULL, "x and amax must not be NULL");
    if (!aligned16(x)) return fail(FP8LIN_ERR_ALIGN, "x must be 16-byte aligned");
    if (!check_arch()) return fail(FP8LIN_ERR_ARCH, "fp8lin kernels are built for sm_100a only");
    cudaError_t e = launch_abs_max((const __nv_bfloat16*)x, ldx, M, K, amax, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "abs-max launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_quantize_activation(const void* x, int64_t ldx, const float* input_scale, void* xq, int64_t M, int64_t K,
                               void* stream) {
    if (M < 0 || K <= 0 || K % 16 != 0) return fail(FP8LIN_ERR_SHAPE, "bad shape M=%lld K=%lld", (long long)M, (long long)K);
    if (M == 0) return FP8LIN_OK;
    if (!x || !input_scale || !xq) return fail(FP8LIN_ERR_NULL, "x, input_scale and xq must not be NULL");
    if (ldx < K || ldx % 8 != 0 || !aligned16(x) || !aligned16(xq)) return fail(FP8LIN_ERR_ALIGN, "x/xq alignment or ldx");
    cudaError_t e = launch_act_quant((const __nv_bfloat16*)x, ldx, input_scale, (unsigned char*)xq, M, K, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "activation quantiser launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

static const char* umma_plan_name(int64_t M, int64_t K, int64_t N, char* buf, size_t size) {
    const UmmaPlan pl = plan_umma(M, K, N, g_tune.umma_bn, g_tune.umma_splits);
    if (pl.tail_tiles) snprintf(buf, size, "umma_w8a8_128x%d_s1+tail%dx%d", pl.bn, pl.tail_tiles, pl.tail_splits);
    else if (pl.narrow_tiles) snprintf(buf, size, "umma_w8a8_128x%d_s1+half%d", pl.bn, pl.narrow_tiles);
    else snprintf(buf, size, "umma_w8a8_128x%d_s%d", pl.bn, pl.splits);
    return buf;
}

const char* fp8lin_variant_name(int scheme, int64_t M, int64_t K, int64_t N) {
    static thread_local char buf[64];
    if (M <= 0 || K <= 0 || N <= 0) return "none";
    const int max_m = g_tune.stream_max_m >= 0 ? g_tune.stream_max_m : kDefaultStreamMaxM;
    if (scheme == FP8LIN_W8A8_STATIC && M > max_m && N % 8 == 0 && pair_rounds_full(M, N)) return "umma_pair_w8a8_256x256";
    if (scheme == FP8LIN_W8A8_STATIC && M > max_m && N % 8 == 0) {
        return umma_plan_name(M, K, N, buf, sizeof(buf));
    }
    if (scheme == FP8LIN_W8A8_STATIC && swap_eligible(M, K, N)) {
        SwapPlan pl = plan_swap(M, K, N, g_tune.swap_splits, swap_prequant(M));
        snprintf(buf, sizeof(buf), "umma_swap_w8a8_m%d_s%d%s", pl.mp, pl.splits, pl.preq ? "_preq" : "");
        return buf;
    }
    if (scheme == FP8LIN_W8A16 && w8a16_umma_eligible(M, K, N, 8, nullptr)) {
        const F16Chunks c = plan_f16_chunks(M, K, N);
        const int64_t full = c.chunk_tiles * kPackTile < N ? c.chunk_tiles * kPackTile : N;
        UmmaPlan pl = plan_umma(M, 2 * pack_kblocks(K) * kPackTile, full, g_tune.umma_bn, g_tune.umma_splits);
        snprintf(buf, sizeof(buf), "umma_w8a16_f16_128x%d_s%d_c%d", pl.bn, pl.splits, (int)c.n_chunks);
        return buf;
    }
    if (scheme == FP8LIN_W8A16 && w8a16_swap_eligible(M, K, N)) {
        SwapPlan pl = plan_swap_w8a16(M, K, N, g_tune.swap_splits);
        snprintf(buf, sizeof(buf), "umma_swap_w8a16_m%d_s%d", pl.mp, pl.splits);
        return buf;
    }
    StreamPlan sp = plan_stream(scheme, M, K, N, g_tune.stream_splits);
    snprintf(buf, sizeof(buf), "stream_mma_%s_m%d_s%d", scheme == FP8LIN_W8A16 ? "w8a16" : "w8a8", sp.mt * 8, sp.splits);
    return buf;
}

const char* fp8lin_kernel_name(int scheme, int64_t M, int64_t K, int64_t N) {
    static thread_local char buf[64];
    if (M > 0 && K > 0 && N > 0) {
        const W8a16PairPlan* p16 = scheme == FP8LIN_W8A16 ? w8a16_pair_route(M, K, N, 8, nullptr) : nullptr;
        const W8a8PairPlan* p8 = scheme == FP8LIN_W8A8_STATIC ? w8a8_pair_route(M, K, N, 8, nullptr) : nullptr;
        if (p16) snprintf(buf, sizeof(buf), "umma_w8a16_pair_256x%d_s%d", p16->tokens, p16->splits);
        else if (p8) snprintf(buf, sizeof(buf), "umma_w8a8_pair_256x%d_s%d%s", p8->tokens, p8->slices, p8->splits > 1 ? "_cluster" : "");
        if (p16 || p8) return buf;
    }
    const int max_m = g_tune.stream_max_m >= 0 ? g_tune.stream_max_m : kDefaultStreamMaxM;
    if (M > max_m && K > 0 && N > 0 && N % 8 == 0 && scheme == FP8LIN_W8A8_STATIC)
        return pair_eligible(M, K, N) ? "umma_pair_w8a8_256x256" : umma_plan_name(M, K, N, buf, sizeof(buf));
    return fp8lin_variant_name(scheme, M, K, N);
}

int fp8lin_set_tuning(const char* knob, int value) {
    if (!knob) return fail(FP8LIN_ERR_NULL, "knob is NULL");
    ++g_tune_version;
    if (!strcmp(knob, "stream_splits")) g_tune.stream_splits = value;
    else if (!strcmp(knob, "stream_max_m")) g_tune.stream_max_m = value;
    else if (!strcmp(knob, "umma_bn")) g_tune.umma_bn = value;
    else if (!strcmp(knob, "umma_splits")) g_tune.umma_splits = value;
    else if (!strcmp(knob, "swap_splits")) g_tune.swap_splits = value;
    else if (!strcmp(knob, "swap_enable")) g_tune.swap_enable = value;
    else if (!strcmp(knob, "swap_min_m")) g_tune.swap_min_m = value;
    else if (!strcmp(knob, "swap_preq_min_m")) g_tune.swap_preq_min_m = value;
    else if (!strcmp(knob, "w8a16_swap_enable")) g_tune.w8a16_swap_enable = value;
    else if (!strcmp(knob, "w8a16_swap_min_m")) g_tune.w8a16_swap_min_m = value;
    else if (!strcmp(knob, "w8a16_umma_min_m")) g_tune.w8a16_umma_min_m = value;
    else if (!strcmp(knob, "w8a16_chunk_mb")) g_tune.w8a16_chunk_mb = value;
    else if (!strcmp(knob, "w8a16_pair")) g_tune.w8a16_pair = value;
    else if (!strcmp(knob, "w8a16_pair_tokens")) g_tune.w8a16_pair_tokens = value;
    else if (!strcmp(knob, "w8a8_pair")) g_tune.w8a8_pair = value;
    else if (!strcmp(knob, "w8a8_pair_tokens")) g_tune.w8a8_pair_tokens = value;
    else if (!strcmp(knob, "w8a8_pair_slices")) g_tune.w8a8_pair_slices = value;
    else if (!strcmp(knob, "w8a8_pair_splits")) g_tune.w8a8_pair_splits = value;
    else if (!strcmp(knob, "w8a16_pair_splits")) g_tune.w8a16_pair_splits = value;
    else if (!strcmp(knob, "umma_pair")) g_tune.umma_pair = value;
    else if (!strcmp(knob, "fuse_quant")) g_tune.fuse_quant = value;
    else if (!strcmp(knob, "quant_lead")) g_tune.quant_lead = value;
    else if (!strcmp(knob, "stream_push")) set_stream_push(value != 0);
    else if (!strcmp(knob, "mlp_decode_fused")) g_tune.mlp_decode_fused = value;
    else if (!strcmp(knob, "moe_fused")) g_tune.moe_fused = value;
    else if (!strcmp(knob, "moe_pair")) g_tune.moe_pair = value;
    else if (!strcmp(knob, "moe_rows_major")) g_tune.moe_rows_major = value;
    else if (!strcmp(knob, "pair_stages")) set_pair_stages(value);
    else if (!strcmp(knob, "pdl")) set_pdl_enabled(value != 0);
    else return fail(FP8LIN_ERR_ARG, "unknown tuning knob '%s'", knob);
    return FP8LIN_OK;
}

// ---- MoE -------------------------------------------------------------------------------------
namespace {
// From this many routed rows on, the rows are gathered and quantised once by a separate pass instead of inside the gate_up GEMM (where every
// channel tile would redo it), if that pass can rank them (moe_share_rows).  Measured (us per block, inside the GEMM / the pass): 64
// experts 2048 -> 1024, 512 rows 90 / 80.7, 1024 rows 122 / 84; 128 experts 2048 -> 768, 1024 rows 128 / 113.5; 512 experts 2048 -> 512, 4096 rows 336 /
// 289.  With hundreds of experts it pays later (512 experts, 512 rows 173 / 180, 1024 rows 230 / 236; 1024 experts 1024 -> 256, 2048 rows
// 163 / 159): up to 5 % that this line leaves there.
constexpr int64_t kMoePrequantRows = 512;
struct MoeWs {
    size_t off_offsets, off_sorted, off_chunks, off_meta, off_inv, off_gu, off_hq, off_xq, total;
};
MoeWs moe_ws_layout(int64_t rows, int E, int64_t H, int64_t I) {
    MoeWs w;
    size_t o = FP8LIN_WS_HEADER_BYTES;
    auto take = [&](size_t bytes) { size_t at = o; o = align_up(o + bytes, 256); return at; };
    w.off_offsets = take((size_t)(E + 1) * 4);
    w.off_sorted = take((size_t)(rows > 0 ? rows : 1) * 4);
    w.off_chunks = take((size_t)(E + rows / 16 + 2) * 16);
    w.off_meta = take(16);
    w.off_inv = take((size_t)(rows > 0 ? rows : 1) * 4);
    w.off_gu = take(g_tune.moe_fused == 0 ? (size_t)rows * 2 * I * 2 : 0);      // bf16 gate_up rows: only the separate pass reads them
    // The activations.  The grouping's counts lie there first: the GEMM that writes activations waits for the pass that reads the counts
    // last, and the counting kernel waits for whatever read the activations of a call before.
    const size_t counts = rows >= kMoePrequantRows ? moe_count_ints(rows, E) * 4 : 0;
    w.off_hq = take((size_t)rows * I > counts ? (size_t)rows * I : counts);
    w.off_xq = take(rows >= kMoePrequantRows ? (size_t)rows * H : 0);
    w.total = o;
    return w;
}
}  // namespace

// Expert batches on CTA pairs (umma_grouped_pair.cu): the most rows of a chunk, 0 = one CTA's kernels.
//   The line: more than 32 rows per expert, of at least kMoePrequantRows.  Measured (us per block in a loop, one CTA / pairs): 60
//   experts 2048 -> 1408, 34 rows each 115 / 105, 68 rows 124.6 / 122.5, 136 rows 180 / 148, 273 rows 278 / 219; 64 experts 1024 -> 512,
//   40 rows 48.8 / 39.6; 8 experts 1024 -> 512, 4096 rows 128 / 120; but 30 experts 1152 -> 1200, 26 rows 41.4 / 43.8.  Up to 128 rows a pair
//   has to have two work items of either projection: 16 experts 2048 -> 1024, 75 rows 36.9 / 38.4 (128 items, 74 pairs); a chunk of more
//   can be cut (8 experts 1024 -> 1408, 175 rows, 88 items 33.4 / 31.0).
//   Nor pairs where one CTA each does the 128 x 256 items of either projection in one round that fills more than two thirds of the chip, with
//   more than 192 rows per expert (one CTA / pairs): 8 experts 1024 -> 512, 450 rows 25.1 / 25.9, 512 rows 25.2 / 27.7, but 600 rows (1.1 rounds)
//   34.8 / 31.1; 4 experts 2048 -> 1024, 500 rows 29.1 / 31.6; 12 experts 1024 -> 512, 300 rows 25.6 / 28.1; 2 experts 3584 -> 1408, 600 rows
//   38.7 / 42.5; 6 experts 1536 -> 640, 500 rows 31.4 / 31.4.  With half of the chip or fewer rows the cuts between pairs pay for more: 8 experts
//   1024 -> 512, 300 rows 24.2 / 22.6, 16 experts (128 items) 160 rows 25.4 / 24.4, 2 experts 2048 -> 2048, 350 rows (96 items) 28.4 / 27.1.
//   The chunk: a busy expert's rows, should the tokens choose at random (mean and three deviations), up to 320.  Above that an expert in two
//   chunks has its weights loaded twice, but items of up to 256 rows lie in tensor memory beside each other, which longer ones do not: up
//   to 320 as long as most experts fit into one chunk (mean and half a deviation, 311 rows; with K of 512 or less, where the epilogues are the
//   longer part, or with gate_up items for less than two thirds of the pairs, where all are cut between groups of rows anyway, nearly all of
//   them: mean and two, 286 rows), 256 beyond.  Time with chunks of up to 320 over that of 256, three routings each:
//       rows per expert         276   284   292   300   308   316   330   480   530   590   640
//       60, 2048 -> 1408       0.87  0.88  0.91  0.90  0.94  0.97  0.99  0.99  0.89  0.98  1.03
//       48, 1280 -> 1280       0.92  0.91  0.93  0.99  0.99  1.01  1.05  1.00  0.96  0.98  1.01
//       16, 2048 -> 1024       0.88  0.89  0.90  0.91  0.92  0.96  1.02  1.01  1.07  1.02  1.00
//       20, 3584 -> 1024       0.98  0.95  0.99  1.00  0.99  1.03  1.07  1.02  1.01  1.03  1.07
//       64, 1536 ->  640       0.95  0.97  0.94  0.96  1.01  0.99  1.04  1.00  0.95  1.00  1.01
//       64, 1024 ->  512       0.95  0.97  1.00  1.00  1.08  1.04  1.06  0.95  0.95  0.98
//        8, 1024 ->  512       0.95  1.05  1.05  1.05  1.01  1.03  1.05  1.00  0.96  0.96  0.97
//   and, four routings, 292 and 300 rows: 8 experts 3584 -> 1408 0.94 0.94; 8, 2048 -> 1280 0.96 0.97; 5, 2048 -> 1408 (55 items of gate_up)
//   0.97 0.97; 4, 2048 -> 1408 (44) 1.00 1.00; 4, 2048 -> 1024 (32) 1.05 1.05; 2, 2048 -> 1408 (22) 1.00 1.01.
//   Shorter chunks leave room for more slots, but below 192 rows that buys nothing.
namespace {
int moe_pair_rows(int64_t rows, int E, int64_t H, int64_t I, const void* out, int64_t ld_out) {
    if (g_tune.moe_pair == 0 || g_tune.moe_fused == 0 || g_tune.moe_rows_major >= 0 || rows < kMoePrequantRows || E > 1024) return 0;
    if (ld_out % 2 != 0 || (reinterpret_cast<uintptr_t>(out) & 3) != 0) return 0;   // (down stores two channels, 4 bytes, at once)
    if (g_tune.moe_pair > 0) return (int)align_up((size_t)(g_tune.moe_pair < kGroupedPairMaxRows ? g_tune.moe_pair : kGroupedPairMaxRows), 32);
    const int64_t avg = (rows + E - 1) / E;
    const int64_t items = E * (pack_ntiles(I) < (pack_ntiles(H) + 1) / 2 ? pack_ntiles(I) : (pack_ntiles(H) + 1) / 2);
    if (avg <= 32 || (avg <= 128 && items < sm_count())) return 0;
    const double mean = (double)avg, deviation = sqrt(mean);
    // chunks of 128 rows (grouped_rows_kernel's), should the tokens choose at random: the mean over four equal parts of that distribution
    double chunks = 0.0;
    for (const double d : {-1.15, -0.32, 0.32, 1.15}) chunks += 0.25 * (double)E * ceil((mean + d * deviation) / 128.0);
    const double gate_up = chunks * (double)pack_ntiles(I), down = chunks * (double)((H + 255) / 256), sms = (double)sm_count();
    if (avg > 192 && I % 128 == 0 && ld_out % 8 == 0 && aligned16(out) && gate_up <= sms && down <= sms && 3.0 * gate_up > 2.0 * sms) return 0;
    const int most = mean + (H <= 512 || I <= 512 || 3 * E * pack_ntiles(I) < 2 * (sm_count() / 2) ? 2.0 : 0.5) * deviation <= kGroupedPairMaxRows ? kGroupedPairMaxRows : 256;
    const int64_t busy = (int64_t)align_up((size_t)(mean + 3.0 * deviation), 32);
    return busy < 192 ? 192 : busy < most ? (int)busy : most;
}
}  // namespace

static int moe_route_impl(const void* logits, int logits_dtype, int64_t ld, int64_t T, int E, int top_k, int renormalize,
                          float* topk_w, void* topk_ids, bool ids_i64, void* stream) {
    if (T < 0 || E <= 0 || E > 1024 || top_k <= 0 || top_k > 32 || top_k > E || ld < E)
        return fail(FP8LIN_ERR_SHAPE, "bad router shape T=%lld E=%d top_k=%d ld=%lld (E <= 1024, top_k <= 32)",
                    (long long)T, E, top_k, (long long)ld);
    if (logits_dtype != 0 && logits_dtype != 1) return fail(FP8LIN_ERR_ARG, "logits_dtype must be 0 (f32) or 1 (bf16)");
    if (T == 0) return FP8LIN_OK;
    if (!logits || !topk_w || !topk_ids) return fail(FP8LIN_ERR_NULL, "logits, topk_w and topk_ids must not be NULL");
    cudaError_t e = launch_moe_route(logits, logits_dtype, ld, (int)T, E, top_k, renormalize, topk_w, topk_ids, ids_i64, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "router launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_moe_route(const void* logits, int logits_dtype, int64_t ld, int64_t T, int E, int top_k, int renormalize,
                     float* topk_w, int32_t* topk_ids, void* stream) {
    return moe_route_impl(logits, logits_dtype, ld, T, E, top_k, renormalize, topk_w, topk_ids, false, stream);
}

int fp8lin_moe_route_i64(const void* logits, int logits_dtype, int64_t ld, int64_t T, int E, int top_k, int renormalize,
                         float* topk_w, int64_t* topk_ids, void* stream) {
    return moe_route_impl(logits, logits_dtype, ld, T, E, top_k, renormalize, topk_w, topk_ids, true, stream);
}

int fp8lin_moe_align(const int32_t* ids, int64_t rows, int E, int chunk_rows, int32_t* expert_offsets, int32_t* sorted_rows,
                     int32_t* chunks, int32_t* meta, void* stream) {
    if (rows < 0 || rows > (1ll << 24) || E <= 0 || E > 3071)
        return fail(FP8LIN_ERR_SHAPE, "bad grouping shape rows=%lld E=%d (E <= 3071)", (long long)rows, E);
    if (chunk_rows != 16 && chunk_rows != 32 && chunk_rows != 64 && chunk_rows != 128)
        return fail(FP8LIN_ERR_ARG, "chunk_rows must be 16, 32, 64 or 128");
    if (!ids || !expert_offsets || !sorted_rows || !chunks || !meta) return fail(FP8LIN_ERR_NULL, "a required pointer is NULL");
    if (!aligned16(chunks)) return fail(FP8LIN_ERR_ALIGN, "chunks must be 16-byte aligned");
    cudaError_t e = launch_moe_align(ids, false, (int)rows, E, chunk_rows, expert_offsets, sorted_rows, (int4*)chunks, meta, nullptr,
                                     (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "row grouping launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

size_t fp8lin_moe_workspace_bytes(int64_t rows, int E, int64_t H, int64_t I) {
    if (rows < 0 || E <= 0 || H <= 0 || I <= 0) return FP8LIN_WS_HEADER_BYTES;
    return moe_ws_layout(rows, E, H, I).total;
}

static int moe_experts_impl(const void* x, int64_t ldx, int x_div, const void* ids, bool ids_i64, const float* topk_w, int64_t rows,
                            const void* w13_packed, const float* w13_scale, const float* w13_input_scale,
                            const void* w2_packed, const float* w2_scale, const float* w2_input_scale,
                            int E, int64_t H, int64_t I, void* out_routed, int64_t ld_out,
                            void* workspace, size_t workspace_bytes, void* stream) {
    // E <= 3071: the row-grouping kernel keeps 4E + 2 counters in 48 KB of shared memory
    if (rows < 0 || E <= 0 || E > 3071 || H <= 0 || I <= 0 || H % 16 != 0 || I % 16 != 0 || x_div <= 0)
        return fail(FP8LIN_ERR_SHAPE, "bad MoE shape rows=%lld E=%d H=%lld I=%lld (E <= 3071; H, I multiples of 16)", (long long)rows, E,
                    (long long)H, (long long)I);
    if (rows == 0) return FP8LIN_OK;
    if (rows > (1ll << 24)) return fail(FP8LIN_ERR_SHAPE, "too many routed rows");
    if (!x || !ids || !topk_w || !w13_packed || !w13_scale || !w13_input_scale || !w2_packed || !w2_scale ||
        !w2_input_scale || !out_routed)
        return fail(FP8LIN_ERR_NULL, "a required MoE pointer is NULL");
    if (ldx < H || ldx % 8 != 0 || ld_out < H || !aligned16(x) || !aligned16(w13_packed) || !aligned16(w2_packed))
        return fail(FP8LIN_ERR_ALIGN, "x / packed weights must be 16-byte aligned, ldx a multiple of 8, ldx and ld_out >= H");
    if (!check_arch()) return fail(FP8LIN_ERR_ARCH, "fp8lin kernels are built for sm_100a only");
    const MoeWs L = moe_ws_layout(rows, E, H, I);
    if (!workspace || workspace_bytes < L.total)
        return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes", L.total);
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char* ws = (unsigned char*)workspace;
    int* offsets = (int*)(ws + L.off_offsets);
    int* sorted = (int*)(ws + L.off_sorted);
    int4* chunks = (int4*)(ws + L.off_chunks);
    int* meta = (int*)(ws + L.off_meta);
    int* inv = (int*)(ws + L.off_inv);
    __nv_bfloat16* gu = (__nv_bfloat16*)(ws + L.off_gu);
    unsigned char* hq = ws + L.off_hq;
    // grouped and quantised by kernels that spread over the chip; else one CTA groups and gate_up quantises the rows it gathers
    const bool spread = rows >= kMoePrequantRows && moe_share_rows(rows, x_div) > 0;
    const int pair_rows = !spread ? 0 : moe_pair_rows(rows, E, H, I, out_routed, ld_out);
    const int mp = pair_rows ? pair_rows : grouped_chunk_rows(rows, E);
    // Few work items whose experts fill 128-row chunks: the rows are the MMA M dimension (umma_grouped_rows.cu), in
    // gate_up where the up channels start at a tile.
    const bool rows_major = spread && !pair_rows && mp == 128 && g_tune.moe_rows_major != 0;
    unsigned char* xq = ws + L.off_xq;
    cudaError_t e = spread ? launch_moe_group_quant((const __nv_bfloat16*)x, ldx, x_div, ids, ids_i64, (int)rows, E, mp, pair_rows != 0, w13_input_scale,
                                                    (int*)hq, sorted, chunks, meta, inv, xq, (int)H, st)
                           : launch_moe_align(ids, ids_i64, (int)rows, E, mp, offsets, sorted, chunks, meta, inv, st);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "row grouping launch: %s", cudaGetErrorString(e));
    const char* why = nullptr;
    GroupedArgs a;
    a.x = (const __nv_bfloat16*)x; a.sorted_rows = sorted; a.chunks = chunks; a.meta = meta; a.w_scale = w13_scale;
    a.input_scale = w13_input_scale; a.topk_w = topk_w; a.out = gu; a.status = (int*)workspace;
    a.ldx = (int)ldx; a.x_div = x_div; a.ld_out = (int)(2 * I); a.N = (int)(2 * I); a.K = (int)H; a.n_tiles = 0; a.kblocks = 0;
    a.scatter = 0;
    // the gate_up GEMM's epilogue applies the activation and writes hq (the separate pass stays for comparison)
    const bool fused_act = g_tune.moe_fused != 0;
    GroupedArgs g = a;
    if (fused_act) { g.N = (int)I; g.hq = hq; g.h_scale = w2_input_scale; g.out = nullptr; }
    if (spread) {
        e = pair_rows ? launch_grouped_pair_w8a8(g, pair_rows, w13_packed, E, xq, rows, st, &why)
          : rows_major && fused_act && I % 128 == 0 ? launch_grouped_rows_w8a8(g, w13_packed, E, xq, rows, st, &why)
                                                    : launch_grouped_w8a8(false, mp, g, w13_packed, E, xq, rows, st, &why);
    } else {
        e = launch_grouped_w8a8(true, mp, g, w13_packed, E, nullptr, 0, st, &why);
    }
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "gate_up grouped GEMM launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
    if (!fused_act) {
        e = launch_silu_mul_quant(gu, w2_input_scale, hq, meta, (int)rows, (int)I, st);
        if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "activation launch: %s", cudaGetErrorString(e));
    }
    a.w_scale = w2_scale; a.input_scale = w2_input_scale; a.out = (__nv_bfloat16*)out_routed; a.ld_out = (int)ld_out;
    a.N = (int)H; a.K = (int)I; a.scatter = 1;
    e = pair_rows ? launch_grouped_pair_w8a8(a, pair_rows, w2_packed, E, hq, rows, st, &why)
      : rows_major && ld_out % 8 == 0 && aligned16(out_routed) ? launch_grouped_rows_w8a8(a, w2_packed, E, hq, rows, st, &why)
                                                               : launch_grouped_w8a8(false, mp, a, w2_packed, E, hq, rows, st, &why);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "down grouped GEMM launch: %s (%s)", cudaGetErrorString(e), why ? why : "");
    return FP8LIN_OK;
}

int fp8lin_moe_experts_w8a8(const void* x, int64_t ldx, int x_div, const int32_t* ids, const float* topk_w, int64_t rows,
                            const void* w13_packed, const float* w13_scale, const float* w13_input_scale,
                            const void* w2_packed, const float* w2_scale, const float* w2_input_scale,
                            int E, int64_t H, int64_t I, void* out_routed, int64_t ld_out,
                            void* workspace, size_t workspace_bytes, void* stream) {
    return moe_experts_impl(x, ldx, x_div, ids, false, topk_w, rows, w13_packed, w13_scale, w13_input_scale, w2_packed, w2_scale, w2_input_scale,
                            E, H, I, out_routed, ld_out, workspace, workspace_bytes, stream);
}

int fp8lin_moe_combine(const void* routed, void* y, int64_t T, int top_k, int64_t H, void* stream) {
    if (T < 0 || top_k <= 0 || H <= 0 || H % 8 != 0) return fail(FP8LIN_ERR_SHAPE, "bad combine shape");
    if (T == 0) return FP8LIN_OK;
    if (!routed || !y) return fail(FP8LIN_ERR_NULL, "routed and y must not be NULL");
    if (!aligned16(routed) || !aligned16(y)) return fail(FP8LIN_ERR_ALIGN, "routed and y must be 16-byte aligned");
    cudaError_t e = launch_moe_combine((const __nv_bfloat16*)routed, nullptr, (__nv_bfloat16*)y, H, (int)T, top_k, (int)H, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "combine launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

// The experts' scratch, then the routed rows that the combine reads.
size_t fp8lin_moe_block_workspace_bytes(int64_t T, int top_k, int E, int64_t H, int64_t I) {
    if (T < 0 || top_k <= 0 || E <= 0 || H <= 0 || I <= 0) return FP8LIN_WS_HEADER_BYTES;
    return moe_ws_layout(T * top_k, E, H, I).total + align_up((size_t)(T * top_k) * H * 2, 256);
}

int fp8lin_moe_block_w8a8(const void* x, int64_t ldx, const void* topk_ids, int ids_are_i64, const float* topk_w, int64_t T, int top_k,
                          const void* w13_packed, const float* w13_scale, const float* w13_input_scale,
                          const void* w2_packed, const float* w2_scale, const float* w2_input_scale,
                          int E, int64_t H, int64_t I, void* y, int64_t ld_y, void* workspace, size_t workspace_bytes, void* stream) {
    if (T < 0 || top_k <= 0 || top_k > 32) return fail(FP8LIN_ERR_SHAPE, "bad MoE shape T=%lld top_k=%d (top_k <= 32)", (long long)T, top_k);
    if (T == 0) return FP8LIN_OK;
    if (!y) return fail(FP8LIN_ERR_NULL, "y must not be NULL");
    if (ld_y < H || ld_y % 8 != 0 || !aligned16(y)) return fail(FP8LIN_ERR_ALIGN, "y must be 16-byte aligned, ld_y a multiple of 8 and at least H");
    const int64_t rows = T * top_k;
    if (rows > (1ll << 24)) return fail(FP8LIN_ERR_SHAPE, "too many routed rows");
    const MoeWs L = moe_ws_layout(rows, E > 0 ? E : 1, H, I);
    if (!workspace || workspace_bytes < fp8lin_moe_block_workspace_bytes(T, top_k, E, H, I))
        return fail(FP8LIN_ERR_WORKSPACE, "workspace too small: need %zu bytes", fp8lin_moe_block_workspace_bytes(T, top_k, E, H, I));
    __nv_bfloat16* routed = (__nv_bfloat16*)((unsigned char*)workspace + L.total);
    int rc = moe_experts_impl(x, ldx, top_k, topk_ids, ids_are_i64 != 0, topk_w, rows, w13_packed, w13_scale, w13_input_scale, w2_packed, w2_scale,
                              w2_input_scale, E, H, I, routed, H, workspace, L.total, stream);
    if (rc != FP8LIN_OK) return rc;
    cudaError_t e = launch_moe_combine(routed, (const int*)((unsigned char*)workspace + L.off_inv), (__nv_bfloat16*)y, ld_y, (int)T, top_k, (int)H,
                                       (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "combine launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_debug_wait_timeout(void* workspace, int64_t limit_us, void* stream) {
    if (!workspace) return fail(FP8LIN_ERR_NULL, "workspace must not be NULL");
    if (limit_us < 1 || limit_us > 100000) return fail(FP8LIN_ERR_ARG, "limit_us must be 1..100000");
    if (!check_arch()) return fail(FP8LIN_ERR_ARCH, "fp8lin kernels are built for sm_100a only");
    // clock64 ticks at the SM clock: at most ~2 GHz, so 2000 cycles per microsecond is an upper bound
    cudaError_t e = launch_wait_timeout_probe((int*)workspace, (long long)limit_us * 2000, nullptr, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "probe launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int64_t fp8lin_debug_moe_share_rows(int64_t rows, int x_div) {
    return rows >= kMoePrequantRows && rows <= (1ll << 24) && x_div > 0 ? moe_share_rows(rows, x_div) : 0;
}

int fp8lin_debug_moe_pair_rows(int64_t rows, int E, int64_t H, int64_t I) {
    return rows > 0 && E > 0 && H > 0 && I > 0 ? moe_pair_rows(rows, E, H, I, nullptr, H) : 0;
}

int fp8lin_debug_silu(const void* g, float* fast, float* divided, int64_t n, void* stream) {
    if (n < 0 || n > (1ll << 30)) return fail(FP8LIN_ERR_SHAPE, "n must be 0..2^30");
    if (n == 0) return FP8LIN_OK;
    if (!g || !fast || !divided) return fail(FP8LIN_ERR_NULL, "g, fast and divided must not be NULL");
    if (!check_arch()) return fail(FP8LIN_ERR_ARCH, "fp8lin kernels are built for sm_100a only");
    cudaError_t e = launch_silu_probe((const __nv_bfloat16*)g, fast, divided, n, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "probe launch: %s", cudaGetErrorString(e));
    return FP8LIN_OK;
}

int fp8lin_read_status(void* workspace, void* stream, int* status_out) {
    if (!workspace || !status_out) return fail(FP8LIN_ERR_NULL, "workspace and status_out must not be NULL");
    cudaStream_t st = (cudaStream_t)stream;
    int v = 0;
    cudaError_t e = cudaMemcpyAsync(&v, workspace, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(FP8LIN_ERR_LAUNCH, "status read: %s", cudaGetErrorString(e));
    *status_out = v;
    if (v != 0) {
        cudaMemsetAsync(workspace, 0, sizeof(int), st);
        cudaStreamSynchronize(st);
        return fail(FP8LIN_ERR_DEVICE, "a kernel gave up a bounded wait (device status 0x%x)", v);
    }
    return FP8LIN_OK;
}

}  // extern "C"
