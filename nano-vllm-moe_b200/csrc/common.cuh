// Shared device helpers for the fp8lin kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fp8lin.h"

namespace fp8lin {

// ---- scratch header ---------------------------------------------------------
// The first FP8LIN_WS_HEADER_BYTES of the caller's scratch.  Everything in it
// is zero between calls: counters are reset by the CTA that consumes them.
constexpr int kWsStatusWords = 64;                                  // word 0 = device status
constexpr int kWsMaxCounters = FP8LIN_WS_HEADER_BYTES / 4 - kWsStatusWords;

struct WsView {
    int* status;          // device status word (0 = ok)
    int* counters;        // kWsMaxCounters split-K arrival counters
    unsigned char* body;  // shape-dependent area, 256-byte aligned
    size_t body_bytes;
};

__host__ __device__ inline WsView ws_view(void* ws, size_t bytes) {
    WsView v;
    v.status = reinterpret_cast<int*>(ws);
    v.counters = reinterpret_cast<int*>(ws) + kWsStatusWords;
    v.body = reinterpret_cast<unsigned char*>(ws) + FP8LIN_WS_HEADER_BYTES;
    v.body_bytes = bytes > FP8LIN_WS_HEADER_BYTES ? bytes - FP8LIN_WS_HEADER_BYTES : 0;
    return v;
}

// device status codes written by kernels that gave up a bounded wait
enum : int { kDevOk = 0, kDevTimeoutFull = 0x101, kDevTimeoutEmpty = 0x102, kDevTimeoutTmemFull = 0x103,
             kDevTimeoutTmemEmpty = 0x104, kDevTimeoutQuant = 0x105, kDevTimeoutPeer = 0x106 };

// A wait that gave up leaves its code in the status word, and in the host's word whose address the header holds (the words
// behind the status: kWsHostWord; 0 = none), which a caller can look at on every call without asking the device.
constexpr int kWsHostWord = 2;
__device__ __forceinline__ void report_status(int* status, int code) {
    atomicExch(status, code);
    volatile int* host = *reinterpret_cast<int* volatile*>(status + kWsHostWord);
    if (host) {
        *host = code;
        __threadfence_system();
    }
}

// ---- packed weight layout ----------------------------------------------------------
// Weights are stored as 128-channel x 128-byte tiles, each tile contiguous (16 KiB),
// tiles of one channel block consecutive along K:
//   byte(n, k) = ((n / 128) * KB + k / 128) * 16384 + (n % 128) * 128 + (k % 128),  KB = ceil(K / 128)
// N and K are zero-padded to multiples of 128.  A CTA that streams a channel block
// reads one long sequential range of HBM, and a tile is exactly one TMA box.
constexpr int kPackTile = 128;
constexpr int kPackTileBytes = kPackTile * kPackTile;
__host__ __device__ inline int64_t pack_kblocks(int64_t K) { return (K + kPackTile - 1) / kPackTile; }
__host__ __device__ inline int64_t pack_ntiles(int64_t N) { return (N + kPackTile - 1) / kPackTile; }
__host__ __device__ inline size_t pack_offset(int64_t n, int64_t k, int64_t KB) {
    return (size_t)((n >> 7) * KB + (k >> 7)) * kPackTileBytes + (size_t)(n & 127) * kPackTile + (size_t)(k & 127);
}

// ---- programmatic dependent launch ------------------------------------------------
// Every kernel lets the next kernel in the stream start launching early
// (pdl_launch_dependents) and, before it touches memory a predecessor may still be
// writing or reading (activations, outputs, scratch, and scales or biases, which a
// caller may have converted just before), waits for the predecessors to finish
// (pdl_wait).  Only packed weights are read before the wait: they are packed once,
// and a kernel that waits for the packing in full is launched behind it.
// Both are no-ops when the launch carries no such dependency.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads of what a kernel in front may have written.  Never through the read-only path (__ldg, ld.global.nc, or a plain read of a
// const __restrict__ parameter): it promises that nobody writes the memory while this kernel runs, which a kernel that starts
// early cannot promise, and the assembler moves such loads in front of the wait.  It did with the rows of the streaming
// kernel when a branch stood in front of the wait: every replay of a graph of single-row steps read stale rows, eager calls
// were too far apart to show it.
__device__ __forceinline__ uint4 ld_dep(const uint4* p) {
    uint4 r;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ float ld_dep(const float* p) {
    float r;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ int ld_dep(const int* p) {
    int r;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ long long ld_dep(const long long* p) {
    long long r;
    asm volatile("ld.global.s64 %0, [%1];" : "=l"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ float ld_dep(const __nv_bfloat16* p) {
    unsigned short r;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(r) : "l"(p));
    return __uint_as_float((uint32_t)r << 16);
}
// ... past L1: what other SMs (or peers) write while the kernel runs
__device__ __forceinline__ uint4 ld_dep_l2(const uint4* p) {
    uint4 r;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ float2 ld_dep_l2(const float2* p) {
    float2 r;
    asm volatile("ld.global.cg.v2.f32 {%0,%1}, [%2];" : "=f"(r.x), "=f"(r.y) : "l"(p) : "memory");
    return r;
}

// ---- small numeric helpers ----------------------------------------------------
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&p);
}

// Two floats -> two e4m3 bytes (lo in bits 0-7), RNE, saturating to +-448.
__device__ __forceinline__ uint16_t cvt_e4m3x2(float lo, float hi) {
    uint16_t r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
    return r;
}

// Two e4m3 bytes -> packed f16x2 (exact).
__device__ __forceinline__ uint32_t cvt_e4m3x2_to_f16x2(uint16_t v) {
    uint32_t r;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(v));
    return r;
}

// Correctly rounded x / s in three instructions, given r = 1/s rounded to nearest
// (Markstein): q0 = x*r is within an ulp, the FMA residual e = x - q0*s is exact,
// and q0 + e*r rounds to the true quotient.  Overflowing or non-finite q0 is
// returned as is (the exact division overflows there too), and so is a zero q0
// (the correction would turn -0 into +0), so the saturating e4m3 conversion
// that follows sees the same value as after a true division.
struct ExactDiv {
    float s, r;
    uint32_t plain_add;        // see quant8_e4m3: 0x8000 - (bf16 bits of the smallest magnitude that needs care), in both halves
    __device__ __forceinline__ explicit ExactDiv(float scale) {
        s = scale;
        r = __fdiv_rn(1.0f, scale);
        const float lim = fminf(1.5e38f, 1.5e38f * scale);
        plain_add = (0x8000u - (__float_as_uint(lim) >> 16)) * 0x00010001u;
    }
    __device__ __forceinline__ float operator()(float x) const {
        const float q0 = x * r;
        const float e = fmaf(-q0, s, x);
        const float q1 = fmaf(e, r, q0);
        return (fabsf(q0) <= 3.0e38f && q0 != 0.f) ? q1 : q0;
    }
};

// g / (1 + e^-g) without the branch of a general division (a slow path that these operands never take, but that keeps the
// chains of a lane's values from overlapping: an epilogue of 16 of them per step was twice as long).  The quotient is refined
// as in ExactDiv from an approximate reciprocal of d = 1 + e^-g; d is in [1, inf]; a zero
// (g = +-0, or d = inf) and an infinite quotient are the answer as they are.  For every bf16 value of g the result equals the division bit for bit.
__device__ __forceinline__ float silu_f32(float g) {
    const float d = 1.f + expf(-g);
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q0 = g * r;
    const float q1 = fmaf(fmaf(-q0, d, g), r, q0);
    return (fabsf(q0) <= 3.0e38f && q0 != 0.f) ? q1 : q0;
}

// Two lanes of fp32 arithmetic per instruction (sm_100).
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint16_t cvt_e4m3x2(uint64_t v) {
    uint16_t r;
    asm("{\n .reg .f32 lo, hi;\n mov.b64 {lo, hi}, %1;\n cvt.rn.satfinite.e4m3x2.f32 %0, hi, lo;\n}" : "=h"(r) : "l"(v));
    return r;
}

// Static activation quantiser for 8 bf16 values (one 16-byte word) -> 8 e4m3 bytes;
// the codes equal the reference's torch path (true division, RNE, clamp to +-448) bit for bit.
//
// The passes that quantise large activations run beside power-limited GEMMs at 1.2 GHz and are bound by instruction issue
// there (five instructions of ExactDiv per element plus its selection).  So the quotients are refined two at a time, and
// what ExactDiv selects per element is handled around them: a zero keeps its sign through an OR on the codes, and values so
// large that q0 could overflow (or infinite, or NaN) send the whole word through ExactDiv.
__device__ __forceinline__ uint2 quant8_e4m3(uint4 v, const ExactDiv& d) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint2 r;
    const uint32_t m = __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
    if (((m + d.plain_add) & 0x80008000u) == 0) {
        const uint64_t rr = pack_f32x2(d.r, d.r), ns = pack_f32x2(-d.s, -d.s);
        uint32_t c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint64_t x = pack_f32x2(bf16_lo(w[i]), bf16_hi(w[i]));
            const uint64_t q0 = mul_f32x2(x, rr);
            c[i] = cvt_e4m3x2(fma_f32x2(fma_f32x2(q0, ns, x), rr, q0));
        }
        r.x = (c[0] | (c[1] << 16)) | (__byte_perm(w[0], w[1], 0x7531) & 0x80808080u);
        r.y = (c[2] | (c[3] << 16)) | (__byte_perm(w[2], w[3], 0x7531) & 0x80808080u);
        return r;
    }
    const uint32_t a = cvt_e4m3x2(d(bf16_lo(v.x)), d(bf16_hi(v.x)));
    const uint32_t b = cvt_e4m3x2(d(bf16_lo(v.y)), d(bf16_hi(v.y)));
    const uint32_t c = cvt_e4m3x2(d(bf16_lo(v.z)), d(bf16_hi(v.z)));
    const uint32_t e = cvt_e4m3x2(d(bf16_lo(v.w)), d(bf16_hi(v.w)));
    r.x = a | (b << 16);
    r.y = c | (e << 16);
    return r;
}

// 8 bf16 -> 8 f16 (RNE; exact for every bf16 inside the f16 normal range).
__device__ __forceinline__ uint4 bf16x8_to_f16x8(uint4 v) {
    uint4 r;
    __half2 h;
    h = __floats2half2_rn(bf16_lo(v.x), bf16_hi(v.x)); r.x = *reinterpret_cast<uint32_t*>(&h);
    h = __floats2half2_rn(bf16_lo(v.y), bf16_hi(v.y)); r.y = *reinterpret_cast<uint32_t*>(&h);
    h = __floats2half2_rn(bf16_lo(v.z), bf16_hi(v.z)); r.z = *reinterpret_cast<uint32_t*>(&h);
    h = __floats2half2_rn(bf16_lo(v.w), bf16_hi(v.w)); r.w = *reinterpret_cast<uint32_t*>(&h);
    return r;
}

// Streaming 16-byte load that does not pollute L1 (weights are read once).  The read-only path: packed weights only.
__device__ __forceinline__ uint4 ld_stream16(const void* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

}  // namespace fp8lin
