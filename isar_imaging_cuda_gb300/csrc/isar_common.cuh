// Common device helpers for the GB300 ISAR imaging kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace isar {

// Constants as the reference defines them (common.cuh:68-73).
constexpr float kPiF = 3.14159265358979f;
constexpr double kPiD = 3.14159265358979;
constexpr double kLightSpeed = 300000000.0;
constexpr int kRangeCut = 512;          // RANGE_NUM_CUT
constexpr int kRangeNumIfdsPc = 4096;   // RANGE_NUM_IFDS_PC (common.cuh:72)
constexpr int kEntropyIters = 120;      // FAST_ENTROPY_ITERATION_NUM
constexpr int kMaxN = 8192;            // largest supported range_num
constexpr int kMaxM = 1024;             // largest supported echo_num
constexpr int kTwN = 16384;             // twiddle table length
// The table is followed by the factors W_{R NS}^{r k} of the transforms' passes
// as [r][k] (k < NS), so that neighbouring lanes (neighbouring k) read
// neighbouring entries: in the table itself they lie r kTwN / (R NS) apart, a
// gather of up to 32 lines per load that held the row transforms up (hrrp
// 1024 x 8192 73 -> 37 us, 512 x 4096 IFDS frame 1175 -> 1155).  Offsets of (NS, R):
constexpr int kTwPass256 = kTwN;                  // (16, 16)
constexpr int kTwPass4096 = kTwPass256 + 256;     // (256, 16)
constexpr int kTwPass512 = kTwPass4096 + 4096;    // (256, 2)
constexpr int kTwPass1024 = kTwPass512 + 512;     // (256, 4)
constexpr int kTwPass2048 = kTwPass1024 + 1024;   // (256, 8)
constexpr int kTwTotal = kTwPass2048 + 2048;

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// conj(a) * b
__device__ __forceinline__ float2 cmulc(float2 a, float2 b)
{
    return make_float2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
// Packed pairs: one issue slot for both components, with the roundings of two
// scalar operations (and never fused with a product).  The block transforms
// issue on 40-57 % of their cycles with the FP32 pipe 28-41 % busy, so fewer
// instructions are what helps: 1024 x 8192 frame 1455 -> 1393 us, 32 learned
// frames 15.98 -> 15.28 ms, hrrp 1024 x 8192 84.5 -> 79.6 us.  Measured on this part,
// of 128 lanes per clock and SM at 16 warps: FADD and FMUL 110, packed 117;
// FFMA of three registers 61-70, packed 79-103.
__device__ __forceinline__ uint64_t f2u(float2 a)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 u2f(uint64_t a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2u(a)), "l"(f2u(b)));
    return u2f(r);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b)
{
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2u(a)), "l"(f2u(b)));
    return u2f(r);
}
// Componentwise product and fused multiply-add of packed pairs.
__device__ __forceinline__ float2 pmul(float2 a, float2 b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2u(a)), "l"(f2u(b)));
    return u2f(r);
}
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(f2u(a)), "l"(f2u(b)), "l"(f2u(c)));
    return u2f(r);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ float cabs2(float2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }

// Phase in cycles held as a 64-bit two's-complement fraction: value / 2^64.
// exp(j*2*pi*frac) from the top 32 bits.
__device__ __forceinline__ float2 cis_frac64(uint64_t ph)
{
    int32_t hi = (int32_t)(ph >> 32);
    float f = (float)hi * 4.656612873077392578125e-10f;   // 2^-31 : f in [-1, 1) half-cycles
    float s, c;
    sincospif(f, &s, &c);
    return make_float2(c, s);
}

__device__ __forceinline__ int bitrev8(int v)
{
    return (int)(__brev((unsigned)v) >> 24);
}

// Argmax key of maxRowsIdxABS (range_alignment.cu:134-168): larger |value|
// first; on equal values the class (index mod 256) with the smaller 8-bit
// reversed number wins (the shared-memory tree keeps its left operand on
// ties), and within a class the smaller index.
struct ArgKey {
    float a;   // |value|
    int i;     // index
};
__device__ __forceinline__ bool argkey_better(const ArgKey& x, const ArgKey& y)
{
    if (x.a != y.a) return x.a > y.a;
    int cx = x.i & 255, cy = y.i & 255;
    if (cx != cy) return bitrev8(cx) < bitrev8(cy);
    return x.i < y.i;
}

__device__ __forceinline__ unsigned float_as_ordered(float f)   // f >= 0
{
    return __float_as_uint(f);
}

}  // namespace isar
