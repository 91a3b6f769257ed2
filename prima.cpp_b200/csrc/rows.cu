// prima.cpp_b200/csrc/rows.cu — norms and embeddings of the layer-list engine with the row in registers (rows.cuh).  Each launcher answers
// cudaErrorNotSupported for rows it does not take (a width that is not a multiple of four or beyond 8192, arrays not at 16 bytes); the callers in norms.cu
// and mixers.cu then run their kernels with an element a thread.
// Bound: the way to L2 and back and the sum's barrier; a kernel's weights are on their way before the kernel in front has ended.
// us, an element a thread and two or three walks over the row / this (alone, from HBM): RMS norm of 2048 rows of 2048 18.4 / 7.5, of one row 6.1 / 3.5; embedding and
// norm of 2048 rows 15.4 / 10.0; layer norm of 1024 rows of 2048 11.6 / 6.3, with residual 13.0 / 8.8.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "layers.h"
#include "mixers.cuh"
#include "rows.cuh"

namespace pb {
namespace {

// y[r] = x[rows[r]] / rms * w
template <int V, typename OT>
__global__ void __launch_bounds__(512) k_rms_rows(const float * x, const int32_t * rows, const float * __restrict__ w, float eps, OT * y,
                                                  int width, int n_rows, int wpr) {
    __shared__ float red[32];
    const RowPlace at(wpr);
    const int r = blockIdx.x * (blockDim.x / (32 * wpr)) + at.row, n4 = width / 4;
    const bool live = r < n_rows;
    float4 wv[V], v[V];
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        wv[i] = c < n4 ? ld4(w, 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_wait();
    const float * in = x + (int64_t) (live && rows ? rows[r] : live ? r : 0) * width;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        v[i] = live && c < n4 ? ld4(in, 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < V; i++) s += squares4(v[i]);
    const float inv = 1.f / sqrtf(row_sum(s, at, red) / (float) width + eps);
    if (!live) return;
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        if (c < n4) put4(y, (int64_t) r * width + 4 * c, make_float4(v[i].x * inv * wv[i].x, v[i].y * inv * wv[i].y, v[i].z * inv * wv[i].z, v[i].w * inv * wv[i].w));
    }
}

// x[t] = table[token] * scale, or its norm with weight w; y[t] = x[t] / rms * wn where y is given
template <int V, typename WT>
__global__ void __launch_bounds__(512) k_embed_rms_rows(const WT * __restrict__ table, int width, const int32_t * __restrict__ tokens, const float * __restrict__ w, float scale,
                                                        float eps, float * __restrict__ x, const float * __restrict__ wn, WT * __restrict__ y, int n_rows, int wpr) {
    __shared__ float red[2][32];
    const RowPlace at(wpr);
    const int r = blockIdx.x * (blockDim.x / (32 * wpr)) + at.row, n4 = width / 4;
    const bool live = r < n_rows;
    const WT * row = table + (int64_t) (live ? tokens[r] : 0) * width;
    float4 v[V];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        v[i] = live && c < n4 ? ld4(row, 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float inv = scale;
    if (w) {
#pragma unroll
        for (int i = 0; i < V; i++) s += squares4(v[i]);
        inv = 1.f / sqrtf(row_sum(s, at, red[0]) / (float) width + eps);
    }
    s = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        if (live && c < n4) {
            const float4 f = w ? ld4(w, 4 * c) : make_float4(1.f, 1.f, 1.f, 1.f);
            v[i] = make_float4(v[i].x * inv * f.x, v[i].y * inv * f.y, v[i].z * inv * f.z, v[i].w * inv * f.w);
            put4(x, (int64_t) r * width + 4 * c, v[i]);
        }
        s += squares4(v[i]);
    }
    if (!y) return;
    const float inv2 = 1.f / sqrtf(row_sum(s, at, red[1]) / (float) width + eps);
    if (!live) return;
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        if (c < n4) {
            const float4 f = ld4(wn, 4 * c);
            put4(y, (int64_t) r * width + 4 * c, make_float4(v[i].x * inv2 * f.x, v[i].y * inv2 * f.y, v[i].z * inv2 * f.z, v[i].w * inv2 * f.w));
        }
    }
}

// RESID: x[r] += mult * (layernorm(m[r]) * w + bias), y[r] = x[r] in the operand type where y is given; else y[r] = layernorm(m[rows[r]]) * w + bias
template <int V, typename OT, bool RESID>
__global__ void __launch_bounds__(512) k_layernorm_rows(const float * m, const int32_t * rows, const float * __restrict__ w, const float * __restrict__ bias,
                                                        float mult, float eps, float * x, OT * y, int width, int n_rows, int wpr) {
    __shared__ float red[2][32];
    const RowPlace at(wpr);
    const int r = blockIdx.x * (blockDim.x / (32 * wpr)) + at.row, n4 = width / 4;
    const bool live = r < n_rows;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v[V], wv[V], bv[V], xv[V];
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        wv[i] = c < n4 ? ld4(w, 4 * c) : zero;
        bv[i] = bias && c < n4 ? ld4(bias, 4 * c) : zero;
    }
    pdl_wait();
    const float * in = m + (int64_t) (live && rows ? rows[r] : live ? r : 0) * width;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        v[i] = live && c < n4 ? ld4(in, 4 * c) : zero;
        if constexpr (RESID) xv[i] = live && c < n4 ? ld4(x, (int64_t) r * width + 4 * c) : zero;
    }
#pragma unroll
    for (int i = 0; i < V; i++) s += sum4(v[i]);
    const float mean = row_sum(s, at, red[0]) / (float) width;
    s = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++)
        if (at.tl + i * at.step < n4) {
            v[i] = make_float4(v[i].x - mean, v[i].y - mean, v[i].z - mean, v[i].w - mean);
            s += squares4(v[i]);
        }
    const float inv = 1.f / sqrtf(row_sum(s, at, red[1]) / (float) width + eps);
    if (!live) return;
#pragma unroll
    for (int i = 0; i < V; i++) {
        const int c = at.tl + i * at.step;
        if (c >= n4) continue;
        float4 o = make_float4(fmaf(v[i].x * inv, wv[i].x, bv[i].x), fmaf(v[i].y * inv, wv[i].y, bv[i].y), fmaf(v[i].z * inv, wv[i].z, bv[i].z), fmaf(v[i].w * inv, wv[i].w, bv[i].w));
        if constexpr (RESID) {
            o = make_float4(fmaf(mult, o.x, xv[i].x), fmaf(mult, o.y, xv[i].y), fmaf(mult, o.z, xv[i].z), fmaf(mult, o.w, xv[i].w));
            put4(x, (int64_t) r * width + 4 * c, o);
            if (y) put4(y, (int64_t) r * width + 4 * c, o);
        } else put4(y, (int64_t) r * width + 4 * c, o);
    }
}

}  // namespace

int launch_rms_rows(const float * x, const int32_t * rows, const float * w, float eps, void * y, int otype, int n_rows, int width, cudaStream_t st) {
    RowShape s;
    if (!row_shape(n_rows, width, s) || !at16(x) || !at16(w) || !at16(y)) return (int) cudaErrorNotSupported;
    auto go = [&](auto kernel, auto * out) { return ck_launch([&] { launch_dep(kernel, dim3(s.grid), dim3(s.threads), 0, st, x, rows, w, eps, out, width, n_rows, s.wpr); }); };
    using B = __nv_bfloat16;
    if (otype == T_BF16) return s.v == 4 ? go(k_rms_rows<4, B>, (B *) y) : go(k_rms_rows<2, B>, (B *) y);
    return s.v == 4 ? go(k_rms_rows<4, float>, (float *) y) : go(k_rms_rows<2, float>, (float *) y);
}
int launch_embed_rms_rows(const void * table, int type, int width, const int32_t * tokens, int n_tokens, const float * w, float scale, float eps, float * x, const float * wn,
                          void * y, cudaStream_t st) {
    RowShape s;
    if (!row_shape(n_tokens, width, s) || !at16(table) || !at16(w) || !at16(x) || !at16(wn) || !at16(y)) return (int) cudaErrorNotSupported;
    auto go = [&](auto kernel, auto * tab) {   // the first kernel of a pass, behind a copy: a plain launch
        using T = std::remove_pointer_t<decltype(tab)>;
        return ck_launch([&] { kernel<<<s.grid, s.threads, 0, st>>>(tab, width, tokens, w, scale, eps, x, wn, (T *) y, n_tokens, s.wpr); });
    };
    using B = __nv_bfloat16;
    if (type == T_BF16) return s.v == 4 ? go(k_embed_rms_rows<4, B>, (B *) table) : go(k_embed_rms_rows<2, B>, (B *) table);
    return s.v == 4 ? go(k_embed_rms_rows<4, float>, (float *) table) : go(k_embed_rms_rows<2, float>, (float *) table);
}
int launch_layernorm_rows(const float * m, const int32_t * rows, const float * w, const float * bias, float mult, float eps, float * x, void * y, int otype, int n_rows, int width,
                          cudaStream_t st) {
    RowShape s;
    if (!row_shape(n_rows, width, s) || !at16(m) || !at16(w) || !at16(bias) || !at16(x) || !at16(y)) return (int) cudaErrorNotSupported;
    auto go = [&](auto kernel, auto * out) { return ck_launch([&] { launch_dep(kernel, dim3(s.grid), dim3(s.threads), 0, st, m, rows, w, bias, mult, eps, x, out, width, n_rows, s.wpr); }); };
    using B = __nv_bfloat16;
    if (otype == T_BF16) {
        if (x) return s.v == 4 ? go(k_layernorm_rows<4, B, true>, (B *) y) : go(k_layernorm_rows<2, B, true>, (B *) y);
        return s.v == 4 ? go(k_layernorm_rows<4, B, false>, (B *) y) : go(k_layernorm_rows<2, B, false>, (B *) y);
    }
    if (x) return s.v == 4 ? go(k_layernorm_rows<4, float, true>, (float *) y) : go(k_layernorm_rows<2, float, true>, (float *) y);
    return s.v == 4 ? go(k_layernorm_rows<4, float, false>, (float *) y) : go(k_layernorm_rows<2, float, false>, (float *) y);
}

}  // namespace pb
