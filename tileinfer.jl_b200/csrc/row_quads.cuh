// Four consecutive elements of a row, widened to 32-bit and rounded once on store: rows of the step through L2 (another kernel may have
// just written them), weights through the read-only path.
#pragma once
#include "common.cuh"

__device__ __forceinline__ float4 load_row4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load_row4(const bf16* p) {
    const uint2 t = __ldcg(reinterpret_cast<const uint2*>(p));
    return make_float4(__uint_as_float(t.x << 16), __uint_as_float(t.x & 0xffff0000u), __uint_as_float(t.y << 16), __uint_as_float(t.y & 0xffff0000u));
}
__device__ __forceinline__ float4 load_weight4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load_weight4(const bf16* p) {
    const uint2 t = __ldg(reinterpret_cast<const uint2*>(p));
    return make_float4(__uint_as_float(t.x << 16), __uint_as_float(t.x & 0xffff0000u), __uint_as_float(t.y << 16), __uint_as_float(t.y & 0xffff0000u));
}
__device__ __forceinline__ void store_row4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store_row4(bf16* p, const float (&v)[4]) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
}
