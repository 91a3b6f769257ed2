// prima.cpp_b200/csrc/rows.cuh — rows of floats in the registers of a few warps: loads, stores and sums for the row-wise steps of the layer-list engine.
// A row of width floats (a multiple of four, 16-byte aligned) is held by `wpr` warps, a thread having the float4s tl, tl + 32 wpr, ... (V at most),
// so that a row is read once, all its loads are in flight together, and a sum costs one barrier (none for a row of one warp).
// What the kernel in front writes comes by pointers without __restrict__ (pdl.h).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mixers.cuh"

namespace pb {
namespace {

__device__ __forceinline__ float4 ld4(const float * p, int64_t i) { return *reinterpret_cast<const float4 *>(p + i); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16 * p, int64_t i) {
    const uint2 r = *reinterpret_cast<const uint2 *>(p + i);
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
}
__device__ __forceinline__ void put4(float * p, int64_t i, float4 v) { *reinterpret_cast<float4 *>(p + i) = v; }
__device__ __forceinline__ void put4(__nv_bfloat16 * p, int64_t i, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2 *>(p + i) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}
__device__ __forceinline__ float sum4(float4 v) { return (v.x + v.y) + (v.z + v.w); }
__device__ __forceinline__ float squares4(float4 v) { return fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w))); }

// this thread's place: its row of the CTA, its first float4 and the step to the next
struct RowPlace {
    int warp, lane, wpr, row, tl, step;
    __device__ __forceinline__ RowPlace(int wpr_) : warp(threadIdx.x >> 5), lane(threadIdx.x & 31), wpr(wpr_), row(warp / wpr_), tl(warp % wpr_ * 32 + lane), step(32 * wpr_) {}
};
// sum over a row's warps, in the warps' order; red: 32 floats of shared memory for this sum alone.  All threads of the CTA take part
__device__ __forceinline__ float row_sum(float v, const RowPlace & at, float * red) {
    v = wsum(v);
    if (at.wpr == 1) return v;
    if (at.lane == 0) red[at.warp] = v;
    __syncthreads();
    const float * mine = red + at.row * at.wpr;
    float s = mine[0];
    for (int i = 1; i < at.wpr; i++) s += mine[i];
    return s;
}

// How rows are dealt to CTAs of at most 512 threads.  Many rows: four float4s a thread, 256 threads a CTA; few rows leave most SMs idle, so a row gets twice the
// threads where they suffice.  us of a pass's two norms, few / many: width 2048 64 rows 6.2 / 7.0, 128 rows 6.5 / 6.9, 512 rows 8.0 / 8.1; width 4096 64 rows 8.1 / 7.8,
// 512 rows 9.2 / 8.2, 2048 rows 16.5 / 14.2; width 1024 the same up to 2048 rows.
constexpr int ROW_WARPS = 16;
struct RowShape { int v, wpr, rows, threads; unsigned grid; };
inline bool row_shape(int n_rows, int width, RowShape & s) {
    if (width <= 0 || width % 4 != 0 || width > 16 * 32 * ROW_WARPS || n_rows <= 0) return false;
    s.v = n_rows >= 128 || width > 8 * 32 * ROW_WARPS ? 4 : 2;
    s.wpr = (width / 4 + 32 * s.v - 1) / (32 * s.v);
    s.rows = n_rows >= 128 && s.wpr < 8 ? 8 / s.wpr : 1;
    s.threads = 32 * s.wpr * s.rows;
    s.grid = (unsigned) ((n_rows + s.rows - 1) / s.rows);
    return true;
}
inline bool at16(const void * p) { return ((uintptr_t) p & 15) == 0; }   // a null pointer, too

}  // namespace
}  // namespace pb
