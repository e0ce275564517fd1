// Four neighbouring channels of a row at a time, for the kernels that keep a token's row in registers.
#pragma once
#include "common.cuh"

__device__ __forceinline__ float4 row_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 row_load4(const bf16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void row_store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void row_store4(bf16* p, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
}
// The K slices of a split product (slice z at p + z * stride) in ascending order, as the stand-alone reduction adds them, eight
// loads in flight; one slice: the finished value.
__device__ __forceinline__ float4 row_sum_slices(const float* p, int splits, long long stride) {
    float4 s = row_load4(p);
    for (int z = 1; z < splits; z += 8) {
        float4 t[8];
#pragma unroll
        for (int u = 0; u < 8; u++) t[u] = z + u < splits ? row_load4(p + (size_t)(z + u) * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 8; u++) s.x += t[u].x, s.y += t[u].y, s.z += t[u].z, s.w += t[u].w;
    }
    return s;
}
inline bool row_odd(const void* p) { return ((uintptr_t)p & 15) != 0; }
// Threads for a row of H channels, four per thread up to 1,024 threads (a function of the width alone: a row's sums have
// one order in every step), and the pieces per thread (1, 2 or 4; 0: too wide).
inline int row_threads(int H) { return H / 4 < 1024 ? (H / 4 + 31) / 32 * 32 : 1024; }
inline int row_pieces(int H) { return H <= 4096 ? 1 : H <= 8192 ? 2 : H <= 16384 ? 4 : 0; }
