// Arithmetic and layout pieces shared by the sweep executors (sweep.cu,
// flow.cu).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace race {

// Rows above kHugeRow entries are summed in segments of kHugeSeg entries,
// one warp each, combined per row in a fixed order.
constexpr int kHugeRow = 512;
constexpr int kHugeSeg = 256;

// The warp that thread `thread` of block `block` belongs to, counted through
// the grid. A warp per row needs 32 threads a row: beyond 2^27 rows their
// number does not fit in 32 bits.
__host__ __device__ constexpr long long warpOf(unsigned block, unsigned threadsPerBlock, unsigned thread) {
    return ((long long)block * threadsPerBlock + thread) >> 5;
}

template <typename VT>
__device__ __forceinline__ float toF(VT v) { return (float)v; }
template <>
__device__ __forceinline__ float toF<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// a*b + c in the accumulation type
__device__ __forceinline__ double mac(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mac(float a, float b, float c) { return fmaf(a, b, c); }

template <typename VT, typename XT>
__device__ __forceinline__ XT ld(const VT *val, int j) {
    if constexpr (sizeof(XT) == 8) return (XT)val[j];
    else return toF<VT>(val[j]);
}

// The four values of an entry group of the SELL copy (16-byte aligned).
__device__ __forceinline__ void groupVals(const double *v, double out[4]) {
    const double2 a = *(const double2 *)v, b = *(const double2 *)(v + 2);
    out[0] = a.x;
    out[1] = a.y;
    out[2] = b.x;
    out[3] = b.y;
}
__device__ __forceinline__ void groupVals(const float *v, float out[4]) {
    const float4 a = *(const float4 *)v;
    out[0] = a.x;
    out[1] = a.y;
    out[2] = a.z;
    out[3] = a.w;
}
__device__ __forceinline__ void groupVals(const __nv_bfloat16 *v, float out[4]) {
    const uint2 a = *(const uint2 *)v;
    out[0] = __uint_as_float(a.x << 16);
    out[1] = __uint_as_float(a.x & 0xffff0000u);
    out[2] = __uint_as_float(a.y << 16);
    out[3] = __uint_as_float(a.y & 0xffff0000u);
}
__device__ __forceinline__ int comp(const int4 &c, int q) { return q == 0 ? c.x : q == 1 ? c.y : q == 2 ? c.z : c.w; }

template <typename XT>
__device__ __forceinline__ XT warpSum(XT v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace race
