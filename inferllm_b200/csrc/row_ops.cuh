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
// The K slices of a split product (slice z at p + z * stride) in ascending order, as the stand-alone reduction adds them, with the
// loads of up to four or nine slices in flight (where there are fewer the last one again: loads under a condition wait for one
// another, which took 0.3 to 0.6 us of a norm's 2 to 3).  A kernel that also takes finished rows has a variant without this: the
// registers that it costs leave room for half the blocks (2,048 rows of 4,096: 17 against 26 us).
template <int N>
__device__ __forceinline__ void row_add_slices(float4& s, const float* p, int z, int splits, long long stride) {
    float4 t[N];
#pragma unroll
    for (int u = 0; u < N; u++) t[u] = row_load4(p + (size_t)min(z + u, splits - 1) * stride);
#pragma unroll
    for (int u = 0; u < N; u++)
        if (z + u < splits) s.x += t[u].x, s.y += t[u].y, s.z += t[u].z, s.w += t[u].w;
}
__device__ __forceinline__ float4 row_sum_slices(const float* p, int splits, long long stride) {
    float4 s = row_load4(p);
    if (splits <= 4) row_add_slices<3>(s, p, 1, splits, stride);
    else
        for (int z = 1; z < splits; z += 8) row_add_slices<8>(s, p, z, splits, stride);
    return s;
}
inline bool row_odd(const void* p) { return ((uintptr_t)p & 15) != 0; }
// Pieces of four channels per thread for a row of H channels (1, 2 or 4; 0: too wide), and the threads, at most 1,024 (functions of
// the width alone: a row's sums have one order in every step).
inline int row_pieces(int H) { return H <= 4096 ? 1 : H <= 8192 ? 2 : H <= 16384 ? 4 : 0; }
inline int row_threads(int H) { return ((H / 4 + row_pieces(H) - 1) / row_pieces(H) + 31) / 32 * 32; }
