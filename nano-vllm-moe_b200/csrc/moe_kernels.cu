// Small kernels around the MoE expert FFN: router, row grouping, activation, combine.
#include "common.cuh"
#include "kernels.h"

namespace fp8lin {

// ---- router ---------------------------------------------------------------------------
// One warp per token: fp32 softmax over the E router logits, then top-k by k rounds of a
// warp arg-max (ties go to the lower expert index), optional renormalisation of the k
// weights.  Same algebra as softmax(dtype=float32) -> topk -> (w / sum w).
// kMaxPerLane: experts per lane (E <= 32 * kMaxPerLane); small expert counts get a short unrolled loop.
template <typename LogitT, typename IdT, int kMaxPerLane>
__global__ void __launch_bounds__(256)
moe_route_kernel(const LogitT* __restrict__ logits, int64_t ld, int T, int E, int top_k, int renormalize,
                 float* __restrict__ out_w, IdT* __restrict__ out_ids) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (token >= T) return;
    float v[kMaxPerLane];
    const LogitT* row = logits + (size_t)token * ld;
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < kMaxPerLane; ++i) {
        const int e = lane + 32 * i;
        v[i] = e < E ? ld_dep(row + e) : -INFINITY;
        mx = fmaxf(mx, v[i]);
    }
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxPerLane; ++i) {
        const int e = lane + 32 * i;
        v[i] = e < E ? expf(v[i] - mx) : 0.f;
        sum += v[i];
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
    for (int i = 0; i < kMaxPerLane; ++i) {
        // a NaN logit makes every probability of the row a NaN: it ranks above all others, as in torch's topk, so that the
        // picks stay experts of this router
        const float pr = v[i] / sum;
        v[i] = (lane + 32 * i) < E ? (pr == pr ? pr : INFINITY) : -1.f;
    }

    float picked_w = 0.f;     // lane j keeps the j-th pick
    int picked_id = 0;
    float wsum = 0.f;
    for (int j = 0; j < top_k; ++j) {
        float best = -2.f;
        int best_e = 0x7fffffff;
#pragma unroll
        for (int i = 0; i < kMaxPerLane; ++i) {
            const int e = lane + 32 * i;
            if (v[i] > best) { best = v[i]; best_e = e; }     // ascending e per lane keeps the lowest index on ties
        }
        for (int o = 16; o; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
            if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
        }
        const float w = best < INFINITY ? best : __int_as_float(0x7fffffff);
        if (lane == j) { picked_w = w; picked_id = best_e; }
        wsum += w;
        if ((best_e & 31) == lane) v[best_e >> 5] = -1.f;     // remove it from the next round
    }
    if (lane < top_k) {
        out_w[(size_t)token * top_k + lane] = renormalize ? picked_w / wsum : picked_w;
        out_ids[(size_t)token * top_k + lane] = picked_id;
    }
}

// Every small kernel of the block is a programmatic dependent launch: the next one's CTAs are resident when the previous
// one ends.
template <typename... Params, typename... Args>
static cudaError_t launch_dependent(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.numAttrs = pdl_attribute(attr);
    cfg.attrs = attr;
    return counted(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
}

template <typename IdT>
static cudaError_t launch_route(const void* logits, int logits_bf16, int64_t ld, int T, int E, int top_k, int renormalize,
                                float* out_w, IdT* out_ids, cudaStream_t stream) {
    if (T == 0) return cudaSuccess;
    const int warps = 8;
    const unsigned grid = (unsigned)((T + warps - 1) / warps);
#define FP8LIN_ROUTE(PER_)                                                                                                 \
    (logits_bf16 ? launch_dependent(moe_route_kernel<__nv_bfloat16, IdT, PER_>, grid, warps * 32, 0, stream,               \
                                    (const __nv_bfloat16*)logits, ld, T, E, top_k, renormalize, out_w, out_ids)            \
                 : launch_dependent(moe_route_kernel<float, IdT, PER_>, grid, warps * 32, 0, stream, (const float*)logits, \
                                    ld, T, E, top_k, renormalize, out_w, out_ids))
    if (E <= 64) return FP8LIN_ROUTE(2);
    if (E <= 256) return FP8LIN_ROUTE(8);
    return FP8LIN_ROUTE(32);
#undef FP8LIN_ROUTE
}

cudaError_t launch_moe_route(const void* logits, int logits_bf16, int64_t ld, int T, int E, int top_k, int renormalize,
                             float* out_w, void* out_ids, bool ids_i64, cudaStream_t stream) {
    return ids_i64 ? launch_route(logits, logits_bf16, ld, T, E, top_k, renormalize, out_w, (long long*)out_ids, stream)
                   : launch_route(logits, logits_bf16, ld, T, E, top_k, renormalize, out_w, (int*)out_ids, stream);
}

// ---- grouping of routed rows by expert ------------------------------------------------------
// One CTA.  counts -> exclusive scan -> scatter.  Also writes the chunk list the grouped GEMM
// walks: every expert's rows are cut into chunks of `chunk_rows`, or (even: moe_place_kernel's) into as few chunks of at most that as
// they fill, of the same size up to the next multiple of 32.
//   sorted_rows[pos]     routed-row index at sorted position pos (rows of one expert are adjacent)
//   expert_offsets[e]    first sorted position of expert e (E+1 entries)
//   chunks[c]            {expert, first sorted position, rows in chunk, 0}
//   meta[0] = number of chunks, meta[1] = number of rows that had a valid local expert id
//   inv[r]               sorted position of routed row r, -1 if its id was not valid (only if inv is given)
// Rows whose id is outside [0, E) are dropped (they belong to another expert-parallel rank).
//
// Every warp counts its own contiguous share of the rows in counters of its own (kWarps x E of them), so that the shared
// memory atomics of a skewed or large batch collide inside a warp only; then the counters become running positions
// (scan over experts, inside an expert over warps) and the warps place their rows.  Against one set of E counters and a
// serial scan by one thread: 5.7 -> 2.8 us for 256 rows of 60 experts.  A single SM's shared memory atomics bound it from a
// few thousand rows on (16384 rows: 14.7 us).

// rows of an expert's chunks but the last, of n rows in all
__device__ __forceinline__ int chunk_size(int n, int chunk_rows, int even) {
    if (!even || n <= 0) return chunk_rows;
    const int k = (n + chunk_rows - 1) / chunk_rows;
    return ((n + k - 1) / k + 31) & ~31;
}
// Exclusive scans of rows, chunks and (even) costs over the experts by one warp or by a block of kWarps, a stretch of the experts
// each, behind what each adds up of the stretches in front; start and cstart have E + 1 entries.  All but start may be left out (null).
template <int kWarps>
__device__ __forceinline__ void scan_experts(const int* total, int E, int chunk_rows, int even, int* start, int* cstart, int* coststart, int* meta) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stretch = (E + 32 * kWarps - 1) / (32 * kWarps) * 32;
    const int first = kWarps == 1 ? 0 : min(E, warp * stretch), last = min(E, first + stretch);
    auto chunks_of = [&](int n, int& c, int& cost) {
        const int size = chunk_size(n, chunk_rows, even);
        c = (n + size - 1) / size;
        cost = even && c ? (c - 1) * grouped_pair_cost(size >> 5) + grouped_pair_cost((n - (c - 1) * size + 31) >> 5) : 0;
    };
    int row_base = 0, chunk_base = 0, cost_base = 0;
    if constexpr (kWarps > 1) {
        if (cstart) {                              // (the divisions once per expert; the scans take them from their own places)
            for (int e = threadIdx.x; e < E; e += 32 * kWarps) {
                int c, cost;
                chunks_of(total[e], c, cost);
                cstart[e] = c;
                if (even) coststart[e] = cost;
            }
            __syncthreads();
        }
        for (int e = lane; e < first; e += 32) {
            row_base += total[e];
            if (cstart) chunk_base += cstart[e];
            if (cstart && even) cost_base += coststart[e];
        }
        row_base = __reduce_add_sync(0xffffffffu, row_base);
        if (cstart) {
            chunk_base = __reduce_add_sync(0xffffffffu, chunk_base);
            cost_base = __reduce_add_sync(0xffffffffu, cost_base);
            __syncthreads();
        }
    }
    for (int e0 = first; e0 < last; e0 += 32) {
        const int n = e0 + lane < last ? total[e0 + lane] : 0;
        int sn = n, c = 0, cost = 0;
        if (cstart && kWarps == 1) chunks_of(n, c, cost);
        if (cstart && kWarps > 1 && e0 + lane < last) {
            c = cstart[e0 + lane];
            if (even) cost = coststart[e0 + lane];
        }
        int sc = c, sw = cost;
        for (int o = 1; o < 32; o <<= 1) {
            const int pn = __shfl_up_sync(0xffffffffu, sn, o);
            if (lane >= o) sn += pn;
            if (cstart) {
                const int pc = __shfl_up_sync(0xffffffffu, sc, o);
                if (lane >= o) sc += pc;
            }
            if (cstart && even) {                  // (no shuffles of zeros in the chain of a decode step's grouping: 0.2 us)
                const int pw = __shfl_up_sync(0xffffffffu, sw, o);
                if (lane >= o) sw += pw;
            }
        }
        if (e0 + lane < last) {
            start[e0 + lane] = row_base + sn - n;
            if (cstart) cstart[e0 + lane] = chunk_base + sc - c;
            if (cstart && even) coststart[e0 + lane] = cost_base + sw - cost;
        }
        row_base += __shfl_sync(0xffffffffu, sn, 31);
        chunk_base += __shfl_sync(0xffffffffu, sc, 31);
        if (cstart && even) cost_base += __shfl_sync(0xffffffffu, sw, 31);
    }
    if (warp == kWarps - 1 && lane == 0 && cstart) {
        start[E] = row_base; cstart[E] = chunk_base;
        meta[0] = chunk_base; meta[1] = row_base;
        if (even) meta[2] = cost_base;
    }
}
__device__ __forceinline__ void write_chunks(const int* total, int E, int chunk_rows, int even, const int* start, const int* cstart,
                                             const int* coststart, int4* chunks) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        const int n = total[e], size = chunk_size(n, chunk_rows, even);
        for (int c = 0, pos = 0; pos < n; ++c, pos += size)
            chunks[cstart[e] + c] = make_int4(e, start[e] + pos, min(size, n - pos), even ? coststart[e] + c * grouped_pair_cost(size >> 5) : 0);
    }
}

template <typename IdT, int kWarps>
__global__ void __launch_bounds__(1024)
moe_align_kernel(const IdT* __restrict__ ids, int rows, int E, int chunk_rows, int* __restrict__ expert_offsets,
                 int* __restrict__ sorted_rows, int4* __restrict__ chunks, int* __restrict__ meta, int* __restrict__ inv) {
    pdl_launch_dependents();
    extern __shared__ int sh[];
    int* count = sh;                       // [kWarps][E]: rows of expert e in warp w's share, then their next position
    int* total = sh + kWarps * E;          // [E]
    int* start = total + E;                // [E + 1]
    int* cstart = start + E + 1;           // [E + 1] chunk prefix
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kWarps * E; i += blockDim.x) count[i] = 0;
    const int share = ((rows + kWarps * 32 - 1) / (kWarps * 32)) * 32;
    const int r0 = min(rows, warp * share), r1 = min(rows, r0 + share);
    constexpr int kBatch = 8;              // ids in flight per lane
    auto load_ids = [&](int r, int end, int* e) {
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const long long id = r + 32 * i < end ? (long long)ld_dep(ids + r + 32 * i) : -1;
            e[i] = id >= 0 && id < E ? (int)id : -1;
        }
    };
    pdl_wait();
    __syncthreads();
    if (warp < kWarps) {
        int* mine = count + warp * E;
        for (int r = r0 + lane; r < r1; r += 32 * kBatch) {
            int e[kBatch];
            load_ids(r, r1, e);
#pragma unroll
            for (int i = 0; i < kBatch; ++i)
                if (e[i] >= 0) atomicAdd(&mine[e[i]], 1);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        int acc = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) { const int c = count[w * E + e]; count[w * E + e] = acc; acc += c; }
        total[e] = acc;
    }
    __syncthreads();
    if (warp == 0) scan_experts<1>(total, E, chunk_rows, 0, start, cstart, nullptr, meta);
    __syncthreads();
    for (int e = threadIdx.x; e <= E; e += blockDim.x) expert_offsets[e] = start[e];
    if (warp < kWarps) {
        int* mine = count + warp * E;
        for (int r = r0 + lane; r < r1; r += 32 * kBatch) {
            int e[kBatch];
            load_ids(r, r1, e);
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int row = r + 32 * i;
                if (row >= r1) break;
                int pos = -1;
                if (e[i] >= 0) {
                    pos = start[e[i]] + atomicAdd(&mine[e[i]], 1);
                    sorted_rows[pos] = row;
                }
                if (inv) inv[row] = pos;
            }
        }
    }
    write_chunks(total, E, chunk_rows, 0, start, cstart, nullptr, chunks);
}

template <typename IdT>
static cudaError_t launch_align(const IdT* ids, int rows, int E, int chunk_rows, int* expert_offsets, int* sorted_rows, int4* chunks,
                                int* meta, int* inv, cudaStream_t stream) {
    // counters per warp: 32 sets where they fit the 48 KB of shared memory (E <= 340), one set beyond (E <= 3071)
    auto smem = [&](int sets) { return (size_t)((sets + 3) * E + 2) * sizeof(int); };
    if (rows > 1024 && smem(32) <= 48 * 1024)
        return launch_dependent(moe_align_kernel<IdT, 32>, 1, 1024, smem(32), stream, ids, rows, E, chunk_rows, expert_offsets, sorted_rows, chunks, meta, inv);
    if (smem(8) <= 48 * 1024)
        return launch_dependent(moe_align_kernel<IdT, 8>, 1, 256, smem(8), stream, ids, rows, E, chunk_rows, expert_offsets, sorted_rows, chunks, meta, inv);
    return launch_dependent(moe_align_kernel<IdT, 1>, 1, 256, smem(1), stream, ids, rows, E, chunk_rows, expert_offsets, sorted_rows, chunks, meta, inv);
}

cudaError_t launch_moe_align(const void* ids, bool ids_i64, int rows, int E, int chunk_rows, int* expert_offsets, int* sorted_rows,
                             int4* chunks, int* meta, int* inv, cudaStream_t stream) {
    return ids_i64 ? launch_align((const long long*)ids, rows, E, chunk_rows, expert_offsets, sorted_rows, chunks, meta, inv, stream)
                   : launch_align((const int*)ids, rows, E, chunk_rows, expert_offsets, sorted_rows, chunks, meta, inv, stream);
}

// (Within an expert the rows land in the arrival order of the atomics.  Every routed row is an
// independent column of the grouped GEMM, so the order does not change a single output bit.)

// ---- group, quantise and place the rows of a large batch ------------------------------------------------------
// From a few hundred rows on the grouping above is one SM's shared-memory atomics (16384 rows: 14.7 us), so it is spread out.
// moe_count_kernel: a block counts its share of the rows by expert and leaves each row's expert and rank inside the share;
// moe_place_kernel: a block sums up what it needs of the counts (every block all of them from L2, 4 bytes per share and expert: 8 KB of
// 16384 rows and 60 experts, 512 KB of 65536 rows and 1024), which gives its rows' places in expert order, and quantises its tokens there:
// xq[place][:] = e4m3(x[r / x_div][:] / scale) for every routed row r with a valid expert.  The grouped GEMM then takes its rows by TMA
// instead of re-quantising them for every channel tile.  A thread converts 16 elements of a token once and stores them to the places of its
// x_div slots: 2 + x_div bytes of traffic per token element.  The first block also writes the chunk list.  Launch times of 16384 rows x
// 2048, 60 experts: 16.4 us on one CTA and 10.2 for the rows before, 3.0 + 16.7 here (6.9 + 12.6 with the last block of the first kernel
// summing up for all); the block of 4096 tokens, 4 of 60 experts, takes 2 % less.
// What grows with the experts is every block's: from 33 experts on the counts of a share are read beside each other by as many threads as
// there are experts, and eight warps scan them.  With a warp for 32 experts at a time and one warp's scan the second kernel took 38 us with 1024
// experts (512 rows; 10 now, one CTA's grouping and the rows 17).  The slots of a token are one thread's, one behind the other; where tokens
// have more than the router gives, blocks share them out (16384 rows x 2048, 60 experts, us per block, all slots one thread's / shared out: 64 of a
// token 165 / 162, 1024 274 / 155, 4096 667 / 157, one token 2250 / 163).
// Blocks in a loop, us, one CTA's grouping and a pass over the rows / here: 60 experts 2048 -> 1408, 512 rows 97.1 / 95.7, 2048 rows
// 115.6 / 103.1; 512 experts 2048 -> 512, 512 rows 183.0 / 179.9, 4096 rows 297.3 / 291.8; 1024 experts 1024 -> 256, 512 rows 89.5 / 89.7, 4096
// rows 190.5 / 181.7.
constexpr int kMoeShares = 128;                    // at most (see moe_count_ints)
constexpr int kRankBits = 18;                      // a row's rank inside its share (see moe_share_rows); the expert (E <= 3071) above it

// all slots of a token lie in the same share
int64_t moe_share_rows(int64_t rows, int x_div) {
    const int64_t tokens = (rows + x_div - 1) / x_div, least = (512 + (int64_t)x_div - 1) / x_div, even = (tokens + kMoeShares - 1) / kMoeShares;
    const int64_t n = (least > even ? least : even) * x_div;
    return n <= 1 << kRankBits ? n : 0;
}

template <typename IdT>
__global__ void __launch_bounds__(512)
moe_count_kernel(const IdT* __restrict__ ids, int rows, int E, int share_rows, int* __restrict__ counts, int* __restrict__ inv) {
    pdl_launch_dependents();
    extern __shared__ int sh[];                    // [E]
    for (int e = threadIdx.x; e < E; e += blockDim.x) sh[e] = 0;
    pdl_wait();
    __syncthreads();
    const int64_t r0 = (int64_t)blockIdx.x * share_rows;
    const int r1 = (int)(r0 + share_rows < rows ? r0 + share_rows : rows);
    for (int r = (int)r0 + (int)threadIdx.x; r < r1; r += blockDim.x) {
        const long long e = (long long)ld_dep(ids + r);
        inv[r] = e >= 0 && e < E ? (int)e << kRankBits | atomicAdd(&sh[e], 1) : -1;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) counts[(size_t)blockIdx.x * E + e] = sh[e];
}

// kMany: the form for more than 32 experts, or more slots of a token than the router gives.  Up to there a warp's lanes hold all experts,
// and fewer loads in flight leave room for five blocks per SM instead of four (48 registers; blocks us, that form / kMany: 8 experts 1024 ->
// 512, 4800 rows, 640 blocks of this kernel, 29.1 / 30.8, 1600 rows 23.0 / 23.3; 32 experts, 9600 rows 42.9 / 44.3, 2240 rows 26.6 / 26.2; 60 experts
// 2048 -> 512, 2400 rows 53.7 / 52.8; 96 experts 1024 -> 512, 3840 rows 46.6 / 44.2; 256 experts 1024 -> 256, 2048 rows 63.3 / 57.3).
template <bool kMany>
__global__ void __launch_bounds__(256, kMany ? 4 : 5)
moe_place_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, int x_div, const int* __restrict__ inv, int rows, const float* __restrict__ input_scale,
                 unsigned char* __restrict__ xq, int H, const int* __restrict__ counts, int shares, int share_tok, int parts, int slot_parts, int E,
                 int chunk_rows, int even, int* __restrict__ sorted_rows, int4* __restrict__ chunks, int* __restrict__ meta) {
    pdl_launch_dependents();
    extern __shared__ int sh[];
    int* before = sh;                              // [E] rows of the expert in the shares in front
    int* total = sh + E;                           // [E]
    int* start = total + E;                        // [E + 1]
    int* cstart = start + E + 1;                   // [E + 1]: the first block only
    int* coststart = cstart + E + 1;               // [E]: there only where `even`
    for (int e = threadIdx.x; e < 2 * E; e += blockDim.x) sh[e] = 0;
    const int block = kMany ? (int)blockIdx.x / slot_parts : (int)blockIdx.x;
    const int share = block / parts, part = block - share * parts;
    // this block's slots of a token (slot_parts > 1: blocks that quantise the same tokens)
    const int slots = kMany ? ((x_div + slot_parts - 1) / slot_parts + 3) & ~3 : x_div;
    const int j_first = kMany ? ((int)blockIdx.x - block * slot_parts) * slots : 0, j_last = kMany ? min(x_div, j_first + slots) : x_div;
    // this block's tokens; it walks whole ones, `per` at a time, so that no element needs a division to find its row
    const int64_t tokens = ((int64_t)rows + x_div - 1) / x_div;
    const int part_tok = (share_tok + parts - 1) / parts;
    const int64_t t_first = (int64_t)share * share_tok + (int64_t)part * part_tok;
    const int64_t t_last = min(min(tokens, (int64_t)(share + 1) * share_tok), t_first + part_tok);
    const int vec_per_row = H / 16;
    const int per = vec_per_row < 256 ? 256 / vec_per_row : 1;
    const int sub = per > 1 ? (int)threadIdx.x / vec_per_row : 0;
    const int c_first = per > 1 ? (int)threadIdx.x - sub * vec_per_row : (int)threadIdx.x, c_step = per > 1 ? vec_per_row : 256;
    const int64_t t_mine = sub < per ? t_first + sub : t_last;
    auto source = [&](int64_t t, int c) { return reinterpret_cast<const uint4*>(x + (size_t)t * ldx + c * 16); };
    pdl_wait();
    uint4 va = make_uint4(0u, 0u, 0u, 0u), vb = va;                        // the first piece is on its way beside the counts
    if (t_mine < t_last && c_first < vec_per_row) {
        va = ld_dep(source(t_mine, c_first));
        vb = ld_dep(source(t_mine, c_first) + 1);
    }
    __syncthreads();
    // threads beside each other sum up experts beside each other, some shares in flight; what is left of the block divides the shares
    constexpr int kFlight = kMany ? 8 : 4;
    const int across = !kMany || E <= 32 ? 32 : E <= 64 ? 64 : E <= 128 ? 128 : 256, groups = 256 / across;
    for (int e = (int)threadIdx.x & (across - 1); e < E; e += across) {
        int all = 0, front = 0;
        for (int b = (int)threadIdx.x / across; b < shares; b += kFlight * groups) {
            int n[kFlight];
#pragma unroll
            for (int i = 0; i < kFlight; ++i) n[i] = b + i * groups < shares ? ld_dep(counts + (size_t)(b + i * groups) * E + e) : 0;
#pragma unroll
            for (int i = 0; i < kFlight; ++i) {
                all += n[i];
                if (b + i * groups < share) front += n[i];
            }
        }
        if (all) atomicAdd(&total[e], all);
        if (front) atomicAdd(&before[e], front);
    }
    __syncthreads();
    const bool first = blockIdx.x == 0;
    if (kMany || threadIdx.x < 32) scan_experts<kMany ? 8 : 1>(total, E, chunk_rows, even, start, first ? cstart : nullptr, first ? coststart : nullptr, meta);
    __syncthreads();
    if (first) write_chunks(total, E, chunk_rows, even, start, cstart, coststart, chunks);

    constexpr int kSlots = kMany ? 4 : 1;                                  // codes in flight
    const ExactDiv div_scale(fmaxf(ld_dep(input_scale), 1e-12f));
    for (int64_t t = t_mine; t < t_last; t += per)
        for (int c = c_first; c < vec_per_row; c += c_step) {
            if (t != t_mine || c != c_first) {
                va = ld_dep(source(t, c));
                vb = ld_dep(source(t, c) + 1);
            }
            const uint2 qa = quant8_e4m3(va, div_scale), qb = quant8_e4m3(vb, div_scale);
            const uint4 o = make_uint4(qa.x, qa.y, qb.x, qb.y);
            for (int j0 = j_first; j0 < j_last; j0 += kSlots) {
                int code[kSlots];
#pragma unroll
                for (int j = 0; j < kSlots; ++j) {
                    const int64_t r = t * x_div + j0 + j;
                    code[j] = (kSlots == 1 || j0 + j < j_last) && r < rows ? ld_dep(inv + r) : -1;
                }
#pragma unroll
                for (int j = 0; j < kSlots; ++j) {
                    if (code[j] < 0) continue;
                    const int e = code[j] >> kRankBits, place = start[e] + before[e] + (code[j] & ((1 << kRankBits) - 1));
                    *reinterpret_cast<uint4*>(xq + (size_t)place * H + c * 16) = o;
                    if (c == 0) sorted_rows[place] = (int)(t * x_div + j0 + j);
                }
            }
        }
}

size_t moe_count_ints(int64_t rows, int E) {
    const int64_t shares = (rows + 511) / 512;     // (a share has 512 rows at least)
    return (size_t)(shares < kMoeShares ? shares : kMoeShares) * E;
}

cudaError_t launch_moe_group_quant(const __nv_bfloat16* x, int64_t ldx, int x_div, const void* ids, bool ids_i64, int rows, int E, int chunk_rows, bool even,
                                   const float* input_scale, int* counts, int* sorted_rows, int4* chunks, int* meta, int* inv, unsigned char* xq, int H,
                                   cudaStream_t stream) {
    const int share_tok = (int)(moe_share_rows(rows, x_div) / x_div), tokens = (rows + x_div - 1) / x_div;
    if (share_tok == 0) return cudaErrorInvalidValue;
    const int shares = (tokens + share_tok - 1) / share_tok;
    const size_t smem = (size_t)E * sizeof(int);
    cudaError_t e = ids_i64 ? launch_dependent(moe_count_kernel<long long>, shares, 512, smem, stream, (const long long*)ids, rows, E, share_tok * x_div, counts, inv)
                            : launch_dependent(moe_count_kernel<int>, shares, 512, smem, stream, (const int*)ids, rows, E, share_tok * x_div, counts, inv);
    if (e != cudaSuccess) return e;
    // parts of a share: about eight blocks per SM in all, but whole turns of a block
    const int vec = H / 16, per = vec < 256 ? 256 / vec : 1;
    int parts = sm_count() * 8 / shares;
    if (parts > (share_tok + per - 1) / per) parts = (share_tok + per - 1) / per;
    if (parts < 1) parts = 1;
    // where that leaves blocks and a token has more slots than the router gives: stretches of at least 64 slots of it
    int slot_parts = x_div > 32 ? sm_count() * 8 / (shares * parts) : 1;
    if (slot_parts > (x_div + 63) / 64) slot_parts = (x_div + 63) / 64;
    if (slot_parts < 1) slot_parts = 1;
    // (E <= 3071, with even chunks <= 1024: 48 KB)
    const auto place = E > 32 || x_div > 32 ? moe_place_kernel<true> : moe_place_kernel<false>;
    return launch_dependent(place, (unsigned)(shares * parts * slot_parts), 256, (size_t)((even ? 5 : 4) * E + 2) * sizeof(int), stream, x, ldx, x_div, inv, rows,
                            input_scale, xq, H, counts, shares, share_tok, parts, slot_parts, E, chunk_rows, even, sorted_rows, chunks, meta);
}

// ---- h = silu(gate) * up, quantised for the down projection ----------------------------------
// gu: bf16 [rows][2I] (gate | up), hq: e4m3 [rows][I].  The reference's experts evaluate
// F.silu(gate) * up as two eager bf16 ops (experts/eager_experts.py:33): silu(gate) is rounded to
// bf16, the product is rounded to bf16 again; that tensor is then divided by the static scale.
__global__ void __launch_bounds__(256)
silu_mul_quant_kernel(const __nv_bfloat16* __restrict__ gu, const float* __restrict__ input_scale,
                      unsigned char* __restrict__ hq, const int* __restrict__ meta, int I) {
    pdl_launch_dependents();
    pdl_wait();
    const int rows = ld_dep(meta + 1);
    const ExactDiv div_scale(fmaxf(ld_dep(input_scale), 1e-12f));
    const int vec_per_row = I / 8;
    const int64_t total = (int64_t)rows * vec_per_row;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / vec_per_row;
        const int c = (int)(i - r * vec_per_row) * 8;
        const uint4 g = ld_dep(reinterpret_cast<const uint4*>(gu + r * 2 * I + c));
        const uint4 u = ld_dep(reinterpret_cast<const uint4*>(gu + r * 2 * I + I + c));
        const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
        uint4 h;
        uint32_t* hw = reinterpret_cast<uint32_t*>(&h);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float g0 = bf16_lo(gw[j]), g1 = bf16_hi(gw[j]);
            const uint32_t sp = pack_bf16x2(silu_f32(g0), silu_f32(g1));
            hw[j] = pack_bf16x2(bf16_lo(sp) * bf16_lo(uw[j]), bf16_hi(sp) * bf16_hi(uw[j]));
        }
        *reinterpret_cast<uint2*>(hq + r * I + c) = quant8_e4m3(h, div_scale);
    }
}

cudaError_t launch_silu_mul_quant(const __nv_bfloat16* gu, const float* input_scale, unsigned char* hq, const int* meta,
                                  int max_rows, int I, cudaStream_t stream) {
    int64_t blocks = ((int64_t)max_rows * (I / 8) + 255) / 256;
    if (blocks > sm_count() * 8) blocks = sm_count() * 8;
    if (blocks < 1) blocks = 1;
    return launch_dependent(silu_mul_quant_kernel, (unsigned)blocks, 256, 0, stream, gu, input_scale, hq, meta, I);
}

// ---- combine: y[t] = bf16( sum over the k routed rows of token t ) ---------------------------
// routed: bf16 [T*k][H] in routed-row order (slot j of token t at row t*k + j), summed in slot order.  inv (optional): a slot
// whose routed row had no valid expert (inv < 0) has not been written and counts as zero.
// A block walks whole rows (no division per element) and a thread has up to four slots' loads in flight.
__global__ void __launch_bounds__(256)
moe_combine_kernel(const __nv_bfloat16* __restrict__ routed, const int* __restrict__ inv, __nv_bfloat16* __restrict__ y, int64_t ld_y, int T,
                   int top_k, int H) {
    pdl_launch_dependents();
    pdl_wait();
    const int vec = H / 8;
    for (int64_t t = blockIdx.x; t < T; t += gridDim.x) {
        const __nv_bfloat16* src = routed + (size_t)t * top_k * H;
        for (int c = threadIdx.x; c < vec; c += blockDim.x) {
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int j0 = 0; j0 < top_k; j0 += 4) {
                uint4 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] = make_uint4(0u, 0u, 0u, 0u);
                    if (j0 + j < top_k && (!inv || ld_dep(inv + t * top_k + j0 + j) >= 0))
                        v[j] = ld_dep(reinterpret_cast<const uint4*>(src + (size_t)(j0 + j) * H + c * 8));
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[0] += bf16_lo(v[j].x); acc[1] += bf16_hi(v[j].x); acc[2] += bf16_lo(v[j].y); acc[3] += bf16_hi(v[j].y);
                    acc[4] += bf16_lo(v[j].z); acc[5] += bf16_hi(v[j].z); acc[6] += bf16_lo(v[j].w); acc[7] += bf16_hi(v[j].w);
                }
            }
            uint4 o;
            o.x = pack_bf16x2(acc[0], acc[1]); o.y = pack_bf16x2(acc[2], acc[3]);
            o.z = pack_bf16x2(acc[4], acc[5]); o.w = pack_bf16x2(acc[6], acc[7]);
            *reinterpret_cast<uint4*>(y + t * ld_y + c * 8) = o;
        }
    }
}

cudaError_t launch_moe_combine(const __nv_bfloat16* routed, const int* inv, __nv_bfloat16* y, int64_t ld_y, int T, int top_k, int H,
                               cudaStream_t stream) {
    if (T == 0) return cudaSuccess;
    const int64_t blocks = T < sm_count() * 16 ? T : sm_count() * 16;
    const unsigned threads = H >= 2048 ? 256 : (H >= 1024 ? 128 : 64);
    return launch_dependent(moe_combine_kernel, (unsigned)blocks, threads, 0, stream, routed, inv, y, ld_y, T, top_k, H);
}

}  // namespace fp8lin
