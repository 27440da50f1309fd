// Row kernels with a row in registers: loads and stores of four consecutive values, and the block a row takes.
#pragma once

#include "common.cuh"

// Four consecutive values at a time, and a row (or group) held in registers between its two passes: every load of a
// thread is asked for before the first is used, so a row costs one trip to memory however wide it is.  Used when
// the width is a multiple of 4 and a thread's share fits RN_MAX_IT groups of four; the plain loops further down serve the rest.
#define RN_MAX_IT 8
__device__ __forceinline__ void rn_load4(const float* p, float (&f)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
__device__ __forceinline__ void rn_load4(const __nv_bfloat16* p, float (&f)[4]) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
__device__ __forceinline__ void rn_load4(const void* p, long long i, int dtype, float (&f)[4]) {
    if (dtype == RDL_BF16) rn_load4((const __nv_bfloat16*)p + i, f); else rn_load4((const float*)p + i, f);
}
__device__ __forceinline__ void rn_store4(float* p, const float (&f)[4]) { *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]); }
__device__ __forceinline__ void rn_store4(__nv_bfloat16* p, const float (&f)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
    uint2 raw;
    raw.x = *reinterpret_cast<const uint32_t*>(&a); raw.y = *reinterpret_cast<const uint32_t*>(&b);
    *reinterpret_cast<uint2*>(p) = raw;
}
// threads of a block whose row is `width` wide: a multiple of 32 that depends on the width alone
static inline int vec_threads(int width) {
    const int groups = width / 4;
    int t = (groups + RN_MAX_IT - 1) / RN_MAX_IT;      // the fewest that keep a thread's share within RN_MAX_IT
    if (t < (groups + 1) / 2) t = (groups + 1) / 2;    // but two groups a thread at most while a block holds them
    t = (t + 31) / 32 * 32;
    return t > 256 ? 256 : (t < 32 ? 32 : t);
}
static inline bool vec_ok(int width, int threads) { return width % 4 == 0 && (width / 4 + threads - 1) / threads <= RN_MAX_IT; }
static inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
// groups of four a thread takes, rounded up to 1, 2, 4 or 8 (the kernels' unrolled depth)
static inline int vec_depth(int width, int threads) {
    const int need = (width / 4 + threads - 1) / threads;
    return need <= 1 ? 1 : (need <= 2 ? 2 : (need <= 4 ? 4 : 8));
}
#define RN_BY_DEPTH(depth, LAUNCH) \
    switch (depth) { case 1: LAUNCH(1); break; case 2: LAUNCH(2); break; case 4: LAUNCH(4); break; default: LAUNCH(8); break; }
