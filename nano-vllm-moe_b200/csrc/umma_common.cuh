// PTX wrappers shared by the tcgen05 kernels: mbarriers with bounded waits, TMA
// loads/stores, TMEM allocation and loads, UMMA descriptors, cluster helpers.
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace fp8lin {

constexpr long long kWaitCycles = 2000000000LL;   // about a second: then a wait gives up

// ---- PTX wrappers --------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// Bounded wait; false = gave up after `limit` clock cycles (status word written).  kTensorMemory: for a barrier that CTAs of
// the cluster arrive on with mbar_arrive_remote; a tcgen05 fence follows.
template <bool kTensorMemory = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* status, int code,
                                          long long limit = kWaitCycles) {
    long long start = -1;
    for (uint32_t it = 0;; ++it) {
        uint32_t done;
        if constexpr (kTensorMemory)
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        else
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if ((it & 0x3ff) == 0x3ff) {
            const long long now = clock64();
            if (start < 0) start = now;
            else if (now - start > limit) { report_status(status, code); return false; }
        }
    }
}
// TMA store of one shared-memory box; elements outside the tensor are not written,
// which is what clips the M and N tails.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- issue from a converged warp ---------------------------------------------------------------------------
// The producer and MMA warps run their loops with all 32 lanes and issue through a predicate that elect.sync gives one lane.
// Inside `if (lane == 0)` the compiler has to treat every address and descriptor as a per-lane value and moves each one to
// the uniform registers these instructions take: measured 92 SM cycles per tcgen05.mma and 160 per pair of commits, against
// 16 and 60 from converged code, which made the issuing thread the limit of every kernel here with small tiles.
// A wait inside such a loop ends in a vote, so that its exit is uniform too.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r));
    return r;
}
// A value that all lanes hold, in a form the compiler knows to be uniform (loaded values are not, shuffled ones neither).
__device__ __forceinline__ int uniform(int v) { return (int)__reduce_or_sync(0xffffffffu, (unsigned)v); }
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, int* status, int code) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, status, code));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t elected, uint32_t bar, uint32_t bytes) {
    asm volatile(
        "{\n .reg .b64 st;\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}"
        ::"r"(bar), "r"(bytes), "r"(elected) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t elected, uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n"
        " @q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n}"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(elected) : "memory");
}
// completion counted on a barrier that may live in the peer CTA (`bar` is a shared::cluster address); the data goes to one CTA
__device__ __forceinline__ void tma_load_2d_pair(uint32_t elected, uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n"
        " @q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n}"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(elected) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t elected, uint32_t bar) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}"
                 ::"r"(bar), "r"(elected) : "memory");
}
// arrives on the barrier at this shared-memory offset in every CTA of `mask` once the pair's MMAs issued so far are done
__device__ __forceinline__ void umma_commit_both(uint32_t elected, uint32_t bar, uint16_t mask) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n"
        " @q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}"
        ::"r"(bar), "h"(mask), "r"(elected) : "memory");
}
#define FP8LIN_UMMA_SS(NAME, GROUP, KIND)                                                                                     \
    __device__ __forceinline__ void NAME(uint32_t elected, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t acc) { \
        asm volatile(                                                                                                         \
            "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"                                        \
            " @q tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], %1, %2, %3, p;\n}"                                     \
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc), "r"(elected) : "memory");                          \
    }
// both operands in shared memory; 32 bytes of K per instruction (32 e4m3 or 16 f16 / bf16)
FP8LIN_UMMA_SS(umma_f8, "1", "f8f6f4")
FP8LIN_UMMA_SS(umma_f16_ss, "1", "f16")
FP8LIN_UMMA_SS(umma_f8_pair, "2", "f8f6f4")
FP8LIN_UMMA_SS(umma_f16_pair, "2", "f16")
#undef FP8LIN_UMMA_SS
// A from tensor memory
__device__ __forceinline__ void umma_f16_ts(uint32_t elected, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc), "r"(elected) : "memory");
}
__device__ __forceinline__ void umma_f16_ts_pair(uint32_t elected, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc), "r"(elected) : "memory");
}

// ---- CTA pairs (cta_group::2): one MMA spans the tensor cores, shared memory and TMEM of two CTAs ----
// Every collective below is executed by the same warp of BOTH CTAs of the pair.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {     // bar: shared::cluster address
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Arrive on a barrier of any CTA of the cluster to hand over tensor memory and nothing else: the tcgen05 accesses are ordered
// by tcgen05.wait and the tcgen05 fences on both sides of the barrier, which take the execution order that a relaxed arrival
// and a relaxed wait at cluster scope give; no other memory is released.  (A release at cluster scope waits until the warp's
// earlier stores have reached L2: over a thousand cycles behind an epilogue's stores.)
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// 32 lanes x 32 columns of fp32 from TMEM (lane i of the warp reads TMEM lane base+i); no wait.
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// cluster helpers (split-K)
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Whole warps come here, and they are brought together first: code in front may have been skipped by a part of the warp, and
// the barrier counts warps.
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    cluster_arrive();
    cluster_wait();
}

// 16 bytes into a CTA of the cluster (dst and bar are shared::cluster addresses of the same CTA); the store is
// asynchronous and counts its bytes on that CTA's barrier when it lands
//
// Split-K hand-overs lay the received sums out as [slice][group of four rows][channel], 16 bytes each: lanes hold channels,
// so an instruction of a warp writes 512 contiguous bytes.  With the four-row groups of a channel side by side each lane's
// 16 bytes travelled alone, and the hand-over was the longest part of a small call: per call back to back, before / after,
// W8A16 64 rows on 3584 -> 3584 10.2 / 9.2 us; W8A8 3584 -> 4608 64 rows 8.6 / 7.6, 2048 -> 2048 one row
// 3.7 / 3.2, 18944 -> 3584 64 rows 15.8 / 14.8.
__device__ __forceinline__ void st_async_v4(uint32_t dst, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(dst), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar) : "memory");
}
__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ float2 ld_shared_f2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

// Tensor memory of a CTA pair, from warp 1 of every CTA.  The allocation and its release reach into the partner CTA, so the
// first waits until every CTA of the cluster runs, and none ends before all are through the second.  Between the two, every
// CTA's mbarriers exist (initialised before the first call); a leader's MMA writes its partner's tensor memory only after rows
// have arrived that the partner's producer loads behind pair_tmem_begin, hence behind its allocation.
//   pair_enter         every CTA of the cluster runs, and its barriers exist: loads may be signalled on them
//   pair_tmem_begin    ... and the tensor memory is there; between the two the producers send the first weights
//   pair_tmem_done     every warp but those of the producers and the MMA issuer, when it has made its last tensor-memory access
//                      (an epilogue warp has then seen the last MMA end, or given up a second ago): arrives in both CTAs
//   pair_tmem_release  warp 1: releases when the warps of both CTAs are done, under the epilogues' last stores
//   pair_leave         nobody ends while its partner may still signal its barriers, or before both have released.  From a
//                      __syncthreads on and by all threads: without it, and with most warps ending in front of a second cluster
//                      barrier, kernels stopped there.
__device__ __forceinline__ void pair_enter() { cluster_sync_all(); }
__device__ __forceinline__ uint32_t pair_tmem_begin(int warp, const uint32_t* s_base, uint32_t cols) {
    if (warp == 1) {
        __syncwarp();
        tmem_alloc_pair(smem_u32(s_base), cols);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    return *s_base;
}
__device__ __forceinline__ void pair_tmem_done(uint32_t bar, uint32_t leader_cta, int lane) {
    tc_fence_before();
    __syncwarp();
    if (lane < 2) mbar_arrive_remote(map_to_cta(bar, leader_cta + (uint32_t)lane));
}
__device__ __forceinline__ void pair_tmem_release(uint32_t bar, uint32_t tmem_base, uint32_t cols, int* status) {
    mbar_wait<true>(bar, 0, status, kDevTimeoutTmemEmpty, 8 * kWaitCycles);      // (the waits it waits for are bounded themselves)
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, cols);
}
__device__ __forceinline__ void pair_leave() {
    __syncthreads();
    cluster_sync_all();
}

// ---- named barriers ------------------------------------------------------------------------------------------
// The form without .aligned: it often follows code that one lane of the warp ran, and whether the warp is together again by
// then is the compiler's choice.
__device__ __forceinline__ void named_sync(int id, int threads) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
// ... with a vote: true in every thread when one of them said so
__device__ __forceinline__ bool named_sync_any(int id, int threads, bool flag) {
    uint32_t any;
    asm volatile(
        "{\n .reg .pred pin, pout;\n setp.ne.b32 pin, %1, 0;\n"
        " barrier.cta.red.or.pred pout, %2, %3, pin;\n selp.u32 %0, 1, 0, pout;\n}"
        : "=r"(any) : "r"(flag ? 1u : 0u), "r"(id), "r"(threads) : "memory");
    return any != 0;
}

// ---- gate_up epilogues: silu(gate) * up, quantised ---------------------------------------------------------------
// What the down projection reads for two rows of a channel, twice kN times: code[j] = two e4m3 codes of h / h_scale, h = bf16(silu(g)
// * u) for the bf16 pairs g[j], u[j].  kTwoRoundings: silu(g) is rounded to bf16 before the product, as the experts' eager
// SiluAndMul does it.  The quotients of silu and of the scale are refined as in silu_f32 and ExactDiv, two lanes an instruction, without what
// those select per value: a gate that could make the exponential overflow (g_max), or an h that is out of the range of quant8_e4m3 (h_max, which
// a NaN in either value reaches; fmaxf passes it by), sends all of the call through them.  (The sign of a zero may differ from theirs, which no product sees.)
// The epilogues run beside MMAs and take their issue slots and power: without the selections and with two lanes an instruction gate_up of
// 4096 tokens, 4 of 60 experts executes 35 million instead of 42 million instructions of a warp, the block takes 2 % less, two 7B decoder
// layers of 1031 rows 0.6 %.
template <int kN, bool kTwoRoundings>
__device__ __forceinline__ void gate_up_codes(const uint32_t (&g)[kN], const uint32_t (&u)[kN], uint32_t (&code)[kN], const ExactDiv& div_h) {
    const uint64_t minus_one = pack_f32x2(-1.f, -1.f), rr = pack_f32x2(div_h.r, div_h.r), ns = pack_f32x2(-div_h.s, -div_h.s);
    float g_max = 0.f;
    uint32_t h_max = 0;
#pragma unroll
    for (int j = 0; j < kN; ++j) {
        const float g0 = bf16_lo(g[j]), g1 = bf16_hi(g[j]);
        g_max = fmaxf(fmaxf(g_max, fabsf(g0)), fabsf(g1));
        const uint64_t gp = pack_f32x2(g0, g1);
        const uint64_t nd = fma_f32x2(pack_f32x2(expf(-g0), expf(-g1)), minus_one, minus_one);          // -(1 + e^-g)
        float n0, n1, r0, r1;
        unpack_f32x2(nd, n0, n1);
        asm("rcp.approx.f32 %0, %1;" : "=f"(r0) : "f"(-n0));
        asm("rcp.approx.f32 %0, %1;" : "=f"(r1) : "f"(-n1));
        const uint64_t r = pack_f32x2(r0, r1), q0 = mul_f32x2(gp, r);
        const uint64_t sv = fma_f32x2(fma_f32x2(q0, nd, gp), r, q0);
        float s0, s1;
        unpack_f32x2(sv, s0, s1);
        uint32_t hv;
        if (kTwoRoundings) {
            const uint32_t sb = pack_bf16x2(s0, s1);
            asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(hv) : "r"(sb), "r"(u[j]));
        } else {
            float h0, h1;
            unpack_f32x2(mul_f32x2(sv, pack_f32x2(bf16_lo(u[j]), bf16_hi(u[j]))), h0, h1);
            hv = pack_bf16x2(h0, h1);
        }
        h_max = __vmaxu2(h_max, hv & 0x7fff7fffu);
        const uint64_t h = pack_f32x2(bf16_lo(hv), bf16_hi(hv)), p0 = mul_f32x2(h, rr);
        code[j] = cvt_e4m3x2(fma_f32x2(fma_f32x2(p0, ns, h), rr, p0));
    }
    if (!(g_max <= 80.f) || ((h_max + div_h.plain_add) & 0x80008000u) != 0) {
#pragma unroll
        for (int j = 0; j < kN; ++j) {
            float s0 = silu_f32(bf16_lo(g[j])), s1 = silu_f32(bf16_hi(g[j]));
            if (kTwoRoundings) {
                const uint32_t sb = pack_bf16x2(s0, s1);
                s0 = bf16_lo(sb);
                s1 = bf16_hi(sb);
            }
            const uint32_t hv = pack_bf16x2(s0 * bf16_lo(u[j]), s1 * bf16_hi(u[j]));
            code[j] = cvt_e4m3x2(div_h(bf16_lo(hv)), div_h(bf16_hi(hv)));
        }
    }
}
// A warp holds kP rows of 32 gate channels, another one the same rows of the up channels (a lane a channel; column pairs of
// rows as bf16x2: lo = rows [0, kP / 2), hi the rest).  Each hands the other half of its values over through swap_buf (kP x 64
// bytes for the two, words [pair][lane], the gate's half in front), the gate warp finishes rows [0, kP / 2), the up warp the
// rest, and code_buf holds e4m3 [row][32 channels] when the call returns (rows that do not exist are computed and not stored by
// the caller).
template <int kP, bool kTwoRoundings>
__device__ __forceinline__ void gate_up_swap(const uint32_t (&lo)[kP / 4], const uint32_t (&hi)[kP / 4], bool up, uint32_t swap_buf,
                                             uint32_t code_buf, int barrier, int lane, const ExactDiv& div_h) {
    constexpr int kH = kP / 4;
#pragma unroll
    for (int j = 0; j < kH; ++j)
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(swap_buf + (up ? 0 : kP * 32) + j * 128 + lane * 4), "r"(up ? lo[j] : hi[j]) : "memory");
    named_sync(barrier, 64);
    uint32_t g[kH], u[kH], code[kH];
#pragma unroll
    for (int j = 0; j < kH; ++j) {
        uint32_t other;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(other) : "r"(swap_buf + (up ? kP * 32 : 0) + j * 128 + lane * 4) : "memory");
        g[j] = up ? other : lo[j];
        u[j] = up ? hi[j] : other;
    }
    gate_up_codes<kH, kTwoRoundings>(g, u, code, div_h);
    const uint32_t code_at = code_buf + (up ? kP * 16 : 0) + lane;
#pragma unroll
    for (int j = 0; j < kH; ++j) {
        asm volatile("st.shared.u8 [%0], %1;" ::"r"(code_at + 2 * j * 32), "r"(code[j] & 0xffu) : "memory");
        asm volatile("st.shared.u8 [%0], %1;" ::"r"(code_at + (2 * j + 1) * 32), "r"(code[j] >> 8) : "memory");
    }
    named_sync(barrier, 64);
}

// ---- K slices of a CTA-pair tile: sums parked in shared memory ------------------------------------------------
// Every CTA of the cluster has its raw sums at smem_base as [group of four tokens][128 channels], 16 bytes each.  This CTA
// finishes channels [c0, c0 + rows) of its pair rank's 128 (n_base: the first of the 128): the up to four slices are added in
// order, then y = bf16(sum * pre * (factor * w_scale[n]) + bias[n]).  After a cluster barrier; the caller keeps the memory alive.
constexpr uint32_t kParkedGroupBytes = 128 * 16u;
__device__ __forceinline__ void finish_parked_band(const UmmaArgs& p, uint32_t smem_base, int splits, int rank, int c0, int rows, int m_valid,
                                                   int n_base, int m_base, float pre, float factor, int threads) {
    const int total = rows * ((m_valid + 3) >> 2);
    for (int i = threadIdx.x; i < total; i += threads) {
        const int c = c0 + i % rows;
        const int mg = i / rows;
        const int n = n_base + c;
        if (n >= p.N) continue;
        const uint32_t local = smem_base + (uint32_t)mg * kParkedGroupBytes + (uint32_t)c * 16u;
        float4 u[4];                                       // all slices' loads go out before the first add
#pragma unroll
        for (int sl = 0; sl < 4; ++sl)
            u[sl] = sl < splits ? ld_cluster_f4(map_to_cta(local, 2u * (uint32_t)sl + (uint32_t)rank)) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 a = u[0];
#pragma unroll
        for (int sl = 1; sl < 4; ++sl) { a.x += u[sl].x; a.y += u[sl].y; a.z += u[sl].z; a.w += u[sl].w; }
        const float ws = factor * ld_dep(p.w_scale + n);
        const float bs = p.bias ? ld_dep(p.bias + n) : 0.f;
        const float o[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (4 * mg + j < m_valid) p.y[(size_t)(m_base + 4 * mg + j) * p.ldy + n] = __float2bfloat16_rn(fmaf(o[j] * pre, ws, bs));
    }
}

// K-major operand tile with 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3ffff) >> 4);   // start address, 16-byte units
    d |= (uint64_t)1 << 16;                    // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                    // descriptor version (Blackwell)
    d |= (uint64_t)2 << 61;                    // SWIZZLE_128B
    return d;
}


// Instruction descriptor: D fp32, A/B formats (0 = e4m3 for kind::f8f6f4; 0 = f16, 1 = bf16 for
// kind::f16), both operands K-major, MMA shape M x N.
__host__ __device__ constexpr uint32_t make_idesc_mn(int m, int n, uint32_t a_fmt, uint32_t b_fmt) {
    return (1u << 4) | (a_fmt << 7) | (b_fmt << 10) | (0u << 15) | (0u << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Opt a kernel in to `bytes` of dynamic shared memory once per device (function attributes are per device).
struct SmemOptIn {
    bool done[64] = {};
};
inline cudaError_t ensure_dynamic_smem(const void* kernel, int bytes, SmemOptIn& state) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && state.done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev >= 0 && dev < 64) state.done[dev] = true;
    return e;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_fn();     // defined in umma_gemm.cu
// How many clusters of `cluster` CTAs of this kernel can be resident at once (cached; when no
// device can be asked, the figure for 148 SMs in 8 GPCs with one CTA per SM).
int max_active_clusters(const void* kernel, int threads, size_t smem_bytes, int cluster);
// 2-D byte tensor [rows][cols] (cols contiguous), box = 128 bytes x box_rows, 128-byte swizzle.
bool encode_u8_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);
// Output map: bf16 [rows][cols] with a row pitch in bytes, box = box_cols x box_rows, swizzle span = the
// box's row length (128 or 64 bytes).
bool encode_out_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes,
                   uint32_t box_cols, uint32_t box_rows = 32);

// ---- activation quantisation inside the large-M GEMM ------------------------------------------------
// The GEMM kernels that take bf16 activations carry kQuantWarps extra warps.  Those warps turn rows
// [row_start, M) of x into e4m3 rows of the scratch matrix xq that the kernel's own TMA producer loads as
// the "A" operand, while the tensor cores work on rows quantised earlier (rows below row_start are
// quantised by a short pass in front of the kernel, so the first round of tiles does not wait).
//
// The work is handed out in units of kQuantRows rows through a ticket counter in global scratch: a warp
// takes the next ticket, converts its rows, and adds one to the "done" counter of the 128-row block the
// rows belong to.  A TMA producer that needs a row block waits (bounded) until that block's counter has
// reached its number of units.  Tickets are only ever taken by warps that are already running, and a warp
// holding a ticket waits for nothing, so the scheme makes progress however many of the grid's CTAs are
// resident at a time.  The last CTA to leave zeroes the counters again (scratch counters are zero between
// calls).  The quantiser warps stay at most `lead` row blocks ahead of the furthest row block any producer has
// started on (the "frontier"): running far ahead would stream all of x and xq through L2 while the GEMM's own
// tiles live there, which measurably slows the GEMM down.  The lead is large enough that a producer never needs
// a block beyond frontier + lead, so the throttle cannot stall the kernel (and a throttle wait that runs out
// simply proceeds).  Layout of ctrl: [0] next ticket, [1] CTAs that have left, [2] frontier, [3 + b] units done
// in row block b.
constexpr int kQuantWarps = 4;
constexpr int kQuantRows = 8;           // rows per unit; divides 128, so a unit lies inside one row block

struct QuantJob {
    const __nv_bfloat16* x;      // bf16 activations [M][ldx]; nullptr = nothing to do (xq arrives complete)
    unsigned char* xq;           // e4m3 [M][K]
    int* ctrl;
    int ldx;
    int row_start;               // multiple of 128
    int lead;                    // row blocks the quantiser may run ahead of the frontier
};
constexpr int kQuantCtrlWords = 3;

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// orders earlier generic-proxy accesses to global memory against later async-proxy (TMA) ones
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Units of the 128-row block `block` that the in-kernel quantiser produces.
__device__ __forceinline__ int quant_units_in_block(const QuantJob& j, int M, int block) {
    const int r0 = max(block * 128, j.row_start);
    const int r1 = min(block * 128 + 128, M);
    return r1 > r0 ? (r1 - r0 + kQuantRows - 1) / kQuantRows : 0;
}

// Producer side: wait until row block `block` of xq is complete.  false = gave up (status written).
__device__ __forceinline__ bool quant_wait_block(const QuantJob& j, int M, int block, int* status) {
    const int need = quant_units_in_block(j, M, block);
    if (need == 0) { atomicMax(j.ctrl + 2, block); return true; }
    atomicMax(j.ctrl + 2, block);          // the frontier moves before the wait: the quantiser may be throttled on it
    const int* flag = j.ctrl + kQuantCtrlWords + block;
    long long start = -1;
    for (uint32_t it = 0;; ++it) {
        if (ld_acquire_gpu(flag) >= need) break;
        if ((it & 0xff) == 0xff) {
            const long long now = clock64();
            if (start < 0) start = now;
            else if (now - start > kWaitCycles) { report_status(status, kDevTimeoutQuant); return false; }
        }
        __nanosleep(64);
    }
    fence_proxy_async_all();       // the rows were written with ordinary stores; the TMA unit reads them next
    return true;
}

// Early, non-blocking look at a row block the producer will need one tile from now: true = already complete
// (completeness is monotonic, so the answer stays valid).  Issued a whole tile ahead, the global round trip of the
// flag load overlaps the tile's loads instead of stalling the producer at the tile boundary.  Also moves the frontier.
__device__ __forceinline__ bool quant_probe_block(const QuantJob& j, int M, int block) {
    atomicMax(j.ctrl + 2, block);
    const int need = quant_units_in_block(j, M, block);
    return need == 0 || ld_acquire_gpu(j.ctrl + kQuantCtrlWords + block) >= need;
}

// One quantiser warp: take units until none are left.
__device__ __forceinline__ void quant_worker(const QuantJob& j, const float* input_scale, int M, int K, int lane) {
    const ExactDiv div(fmaxf(ld_dep(input_scale), 1e-12f));
    const int total_units = M > j.row_start ? (M - j.row_start + kQuantRows - 1) / kQuantRows : 0;
    const int vec_per_row = K >> 4;
    for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(j.ctrl, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= total_units) break;
        const int row0 = j.row_start + u * kQuantRows;
        const int rows = min(kQuantRows, M - row0);
        if ((row0 >> 7) > ld_acquire_gpu(j.ctrl + 2) + j.lead) {          // too far ahead of the GEMM: hold back
            const long long t0 = clock64();
            while ((row0 >> 7) > ld_acquire_gpu(j.ctrl + 2) + j.lead && clock64() - t0 < kWaitCycles) __nanosleep(256);
        }
        // four rows per step: eight 16-byte loads in flight per lane.  The quantiser is latency-bound (a few
        // warps per SM), and it has to keep up with the rate at which the GEMM consumes rows.
        for (int r = 0; r < rows; r += 4) {
            const __nv_bfloat16* src[4];
            unsigned char* dst[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int rr = min(r + q, rows - 1);                   // a short tail re-reads the last row (not stored)
                src[q] = j.x + (size_t)(row0 + rr) * j.ldx;
                dst[q] = j.xq + (size_t)(row0 + rr) * K;
            }
            for (int v = lane; v < vec_per_row; v += 32) {
                uint4 a[4][2];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    a[q][0] = ld_dep(reinterpret_cast<const uint4*>(src[q] + v * 16));
                    a[q][1] = ld_dep(reinterpret_cast<const uint4*>(src[q] + v * 16 + 8));
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (r + q < rows) {
                        const uint2 q0 = quant8_e4m3(a[q][0], div), q1 = quant8_e4m3(a[q][1], div);
                        *reinterpret_cast<uint4*>(dst[q] + v * 16) = make_uint4(q0.x, q0.y, q1.x, q1.y);
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) {
            fence_proxy_async_all();
            __threadfence();
            atomicAdd(j.ctrl + kQuantCtrlWords + (row0 >> 7), 1);
        }
    }
}

// Every CTA calls this once all its warps are done with the counters (after its last __syncthreads):
// the last one to arrive zeroes them for the next call.
__device__ __forceinline__ void quant_ctrl_release(const QuantJob& j, int M) {
    __threadfence();
    const int left = atomicAdd(j.ctrl + 1, 1);
    if (left == (int)gridDim.x - 1) {
        const int blocks = (M + 127) >> 7;
        for (int b = 0; b < blocks; ++b) j.ctrl[kQuantCtrlWords + b] = 0;
        j.ctrl[0] = 0;
        j.ctrl[2] = 0;
        __threadfence();
        j.ctrl[1] = 0;
    }
}

// Destinations of a GEMM epilogue's TMA stores (all describe a bf16 [M][N] matrix of the same shape).
struct OutMaps {
    CUtensorMap m[8];
    int n;
    // 0: every output box is stored to all n destinations.  > 0 (a multiple of 32): destination d receives only the
    // rows [d * band_rows, (d + 1) * band_rows) of the result, at row (r - d * band_rows) of its matrix: the
    // reduce-scatter form of a row-parallel linear, where rank d sums the bands it receives.
    int band_rows;
};

// Store one staged 32-row box whose first row is `row0` of the result to its destination(s).
__device__ __forceinline__ void store_box(const OutMaps& outs, uint32_t box, int col0, int row0) {
    if (outs.band_rows > 0) {
        const int d = row0 / outs.band_rows;
        if (d < outs.n) tma_store_2d(&outs.m[d], box, col0, row0 - d * outs.band_rows);
        else asm volatile("cp.async.bulk.commit_group;" ::: "memory");      // keep the group count per box uniform
        return;
    }
    for (int d = 0; d < outs.n; ++d) tma_store_2d(&outs.m[d], box, col0, row0);
}

// 16 consecutive TMEM columns of this lane -> 16 registers; no wait
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr) : "memory");
}

}  // namespace fp8lin
