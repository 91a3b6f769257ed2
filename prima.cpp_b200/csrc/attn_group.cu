// prima.cpp_b200/csrc/attn_group.cu — decode attention of the engine's per-token path over the f16 cache (row-major K and V, cell == position): rope(q),
// rope(k), cache store, softmax and the quantized activation of the output product in one launch.  The arithmetic is k_attn2's (ops.cu: FA-off
// numerics of the CPU backend, f16-rounded q and probabilities, fp32 sums); the work is laid out for contexts of more than a few cells.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>

#include "launch.h"
#include "quantize.cuh"
#include "rope.cuh"

namespace pb {
namespace {

// One cluster per kv head: its CTAs share the cells in equal consecutive parts and each serves all G query heads of the group, so that a cell is read
// once (one CTA per query head read it G times and walked all of it alone: 24 us a launch at 1000 cells, 32 heads over 8).  Up to 128 cells of a part are on
// their way before the kernel in front has ended; the parts agree on each head's largest score and sum through distributed shared memory, CTA r adds
// super-block r of the group's output in the parts' order and quantizes it.  Buffers of 64 cells twice for K and V: with 70 KB an SM holds this
// kernel beside a CTA of the products around it, whose first weights then travel meanwhile (135 KB and the whole SM cost a short context 6 us a layer).
// Bound: a chain of small steps (load, rope, scores, two exchanges, values, join).
// 24 -> 8 us a launch at 1000 cells.
constexpr int AG_THREADS = 512, AG_WARPS = 16, AG_CHUNK = 64, AG_BUFS = 2, AG_MAX_SPLIT = 8;

template <int G> struct __align__(128) AgSmem {   // behind it: scores [cell of the part][G]
    __align__(128) __half kbuf[AG_BUFS][AG_CHUNK][128];
    __align__(128) __half vbuf[AG_BUFS][AG_CHUNK][128];   // both buffers, read out, take the warps' partial sums [AG_WARPS][G][128]
    uint64_t kbar[AG_BUFS], vbar[AG_BUFS];
    double x_sum[G];               // what the cluster's other CTAs read: this part's sums of exponentials, largest scores and weighed values
    float x_max[G];
    __align__(16) float o_s[G][128];
    double s_redd[AG_WARPS];
    float s_red[AG_WARPS];
    volatile int aborted;          // wait watchdog (common.cuh)
    __align__(16) float q_s[G][128];
    __align__(16) float cs[64][2];
    __align__(16) __half k_s[128];
    __align__(16) __half v_s[128];
};

struct AgParams {
    const float * q; const float * k; const float * v;   // this token's projections (f32, before the rotation)
    __half * kc; __half * vc;     // caches [cell][n_head_kv * 128]
    float * out;                  // [n_head * 128]
    ActQ outq;                    // q8_K of out
    int n_head_kv, splits;
    const int32_t * pos_dev;
    RopeParams rp;
    const float * freq_factors;
    float scale;
    int * abort_flag;
};

__device__ __forceinline__ void ag_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t ag_remote(const void * local, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(local)), "r"(rank));
    return r;
}
__device__ __forceinline__ float ag_ld_f32(const float * local, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ag_remote(local, rank)) : "memory");
    return v;
}
__device__ __forceinline__ void ag_ld_f32x4(const float * local, int rank, float * v) {
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(ag_remote(local, rank)) : "memory");
}
__device__ __forceinline__ double ag_ld_f64(const double * local, int rank) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(ag_remote(local, rank)) : "memory");
    return v;
}
// cells [c * AG_CHUNK, ...) of a part that starts at `cache`; the barrier fires when every thread's copies have landed
__device__ __forceinline__ void ag_issue(__half (*dst)[128], const __half * cache, int64_t row, int c, int ncell, uint64_t * bar) {
    const int r0 = c * AG_CHUNK, pieces = min(AG_CHUNK, ncell - r0) * 16;
    for (int i = threadIdx.x; i < pieces; i += AG_THREADS) {
        const int r = i >> 4, p = i & 15;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&dst[r][p * 8])), "l"(cache + (int64_t) (r0 + r) * row + p * 8) : "memory");
    }
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void ag_row4(const __half * row, int lane, float (&f)[4]) {
    const uint2 raw = *reinterpret_cast<const uint2 *>(row + 4 * lane);
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&raw.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&raw.y));
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}

template <int G>
__global__ void __launch_bounds__(AG_THREADS, 1) k_attn_group(const __grid_constant__ AgParams P) {
    constexpr int D = 128;
    extern __shared__ __align__(128) uint8_t ag_raw[];
    AgSmem<G> * sm = reinterpret_cast<AgSmem<G> *>(ag_raw);
    float * S = reinterpret_cast<float *>(ag_raw + sizeof(AgSmem<G>));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int part = blockIdx.x % P.splits, hk = blockIdx.x / P.splits;
    const int64_t EK = (int64_t) P.n_head_kv * D;
    if (tid == 0) {
#pragma unroll
        for (int b = 0; b < AG_BUFS; b++) { mbar_init(&sm->kbar[b], AG_THREADS); mbar_init(&sm->vbar[b], AG_THREADS); }
        sm->aborted = 0;
        mbar_fence_init();
    }
    __syncthreads();
    pdl_trigger();
    // ---- independent of the product in front: the position (written before this token's first kernel), cache cells of earlier tokens
    const int pos = *P.pos_dev, all = pos + 1;
    // a context of one chunk needs no exchange: the first CTA of the cluster takes it, the others leave (exited threads take no part in
    // the cluster's barriers)
    const int splits = all <= AG_CHUNK ? 1 : P.splits;
    if (part >= splits) return;
    const int per = (all + splits - 1) / splits, cell0 = min(part * per, all), ncell = min(per, all - cell0);   // the last parts may have no cell
    const int fresh = pos - cell0;                        // this token's cell, taken from shared memory; < ncell in the last part that has cells only
    const int nchunks = (ncell + AG_CHUNK - 1) / AG_CHUNK;
    const __half * kc = P.kc + (int64_t) cell0 * EK + hk * D, * vc = P.vc + (int64_t) cell0 * EK + hk * D;
#pragma unroll
    for (int c = 0; c < AG_BUFS; c++)
        if (c < nchunks) ag_issue(sm->kbuf[c], kc, EK, c, ncell, &sm->kbar[c]);
#pragma unroll
    for (int c = 0; c < AG_BUFS; c++)
        if (c < nchunks) ag_issue(sm->vbuf[c], vc, EK, c, ncell, &sm->vbar[c]);
    const RopeParams & rp = P.rp;
    const int half_dims = rp.n_dims / 2;
    const bool neox = rp.mode & 2;
    if (tid < 64 && tid < half_dims) {
        float c, s;
        rope_cos_sin(rp, pos, tid, P.freq_factors, c, s);
        sm->cs[tid][0] = c; sm->cs[tid][1] = s;
    }
    __syncthreads();
    pdl_wait();
    // ---- this token's rows: the group's queries, the key (rotated) and the value, rounded as the cache stores them
    for (int i = tid; i < (G + 2) * 64; i += AG_THREADS) {
        const int r = i >> 6, pair = i & 63;
        if (r > G) {                                      // value: two entries a thread
            const float2 x = __ldcg(reinterpret_cast<const float2 *>(P.v + (int64_t) hk * D) + pair);
            *reinterpret_cast<__half2 *>(sm->v_s + 2 * pair) = __floats2half2_rn(x.x, x.y);
            continue;
        }
        const float * src = r < G ? P.q + (int64_t) (hk * G + r) * D : P.k + (int64_t) hk * D;
        auto keep = [&](int j, float y) {
            const __half h = __float2half_rn(y);
            if (r < G) sm->q_s[r][j] = __half2float(h);
            else sm->k_s[j] = h;
        };
        if (pair < half_dims) {
            const int i0 = neox ? pair : 2 * pair, i1 = neox ? pair + half_dims : 2 * pair + 1;
            float y0, y1;
            rope_rotate(__ldcg(src + i0), __ldcg(src + i1), sm->cs[pair][0], sm->cs[pair][1], y0, y1);
            keep(i0, y0);
            keep(i1, y1);
        }
        for (int j = rp.n_dims + pair; j < D; j += 64) keep(j, __ldcg(src + j));   // the tail that is not rotated
    }
    __syncthreads();
    if (part == 0 && warp == 0) {                         // publish the fresh row; every CTA reads it from its own shared memory
        const int64_t at = (int64_t) pos * EK + hk * D + 4 * lane;
        *reinterpret_cast<uint2 *>(P.kc + at) = *reinterpret_cast<const uint2 *>(sm->k_s + 4 * lane);
        *reinterpret_cast<uint2 *>(P.vc + at) = *reinterpret_cast<const uint2 *>(sm->v_s + 4 * lane);
    }
    // ---- scores (soft_max_ext: the dot times the scale): a warp takes a cell for all heads of the group, a lane four entries of it
    float q[G][4];
#pragma unroll
    for (int g = 0; g < G; g++) *reinterpret_cast<float4 *>(q[g]) = *reinterpret_cast<const float4 *>(&sm->q_s[g][4 * lane]);
    for (int c = 0; c < nchunks; c++) {
        const int b = c % AG_BUFS, r0 = c * AG_CHUNK, nrows = min(AG_CHUNK, ncell - r0);
        mbar_wait(&sm->kbar[b], (uint32_t) ((c / AG_BUFS) & 1), &sm->aborted, P.abort_flag);
        for (int r = warp; r < nrows; r += AG_WARPS) {
            float kf[4], v[G];
            ag_row4(r0 + r == fresh ? sm->k_s : sm->kbuf[b][r], lane, kf);
#pragma unroll
            for (int g = 0; g < G; g++) v[g] = fmaf(kf[3], q[g][3], fmaf(kf[2], q[g][2], fmaf(kf[1], q[g][1], kf[0] * q[g][0])));
            // the G sums over the lanes together: each halving of the lanes halves the values a lane goes on with (the order of a sum is that of warp_sum)
            int head = 0;
#pragma unroll
            for (int o = 16, n = G; o > 0; o >>= 1) {
                if (n > 1) {
                    n >>= 1;
                    const bool up = lane & o;
#pragma unroll
                    for (int i = 0; i < n; i++) {
                        const float send = up ? v[i] : v[i + n], mine = up ? v[i + n] : v[i];
                        v[i] = mine + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                    if (up) head += n;
                } else v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            }
            if ((lane & (32 / G - 1)) == 0) S[(r0 + r) * G + head] = __fmul_rn(v[0], P.scale);
        }
        if (c + AG_BUFS < nchunks) {
            __syncthreads();                              // every warp is done with this buffer
            ag_issue(sm->kbuf[b], kc, EK, c + AG_BUFS, ncell, &sm->kbar[b]);
        }
    }
    __syncthreads();
    // ---- softmax (max, expf, double sum, p = e * float(1 / sum)): warps g, g + G, ... hold head g
    const int g = warp % G, first = warp / G * 32 + lane, step = AG_WARPS / G * 32;
    float m = -INFINITY;
    for (int p = first; p < ncell; p += step) m = fmaxf(m, S[p * G + g]);
    m = warp_max(m);
    if (lane == 0) sm->s_red[warp] = m;
    __syncthreads();
    if (tid < G) {
        float t = sm->s_red[tid];
        for (int w = tid + G; w < AG_WARPS; w += G) t = fmaxf(t, sm->s_red[w]);
        sm->x_max[tid] = t;
    }
    if (splits > 1) ag_cluster_sync(); else __syncthreads();
    const float mx = warp_max(lane < splits ? ag_ld_f32(&sm->x_max[g], lane) : -INFINITY);
    double dsum = 0.0;
    for (int p = first; p < ncell; p += step) {
        const float e = expf(__fsub_rn(S[p * G + g], mx));
        S[p * G + g] = e;
        dsum += (double) e;
    }
    dsum = warp_sum_d(dsum);
    if (lane == 0) sm->s_redd[warp] = dsum;
    __syncthreads();
    if (tid < G) {
        double t = sm->s_redd[tid];
        for (int w = tid + G; w < AG_WARPS; w += G) t += sm->s_redd[w];
        sm->x_sum[tid] = t;
    }
    if (splits > 1) ag_cluster_sync(); else __syncthreads();
    {
        const double mine = lane < splits ? ag_ld_f64(&sm->x_sum[g], lane) : 0.0;
        double t = 0.0;
        for (int i = 0; i < splits; i++) t += __shfl_sync(0xffffffffu, mine, i);
        const float inv = (float) (1.0 / t);
        for (int p = first; p < ncell; p += step) S[p * G + g] = __half2float(__float2half_rn(__fmul_rn(S[p * G + g], inv)));   // f16-rounded probabilities
    }
    __syncthreads();
    // ---- values: a lane owns four entries, the warps share the cells
    float acc[G][4];
#pragma unroll
    for (int i = 0; i < G; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    for (int c = 0; c < nchunks; c++) {
        const int b = c % AG_BUFS, r0 = c * AG_CHUNK, nrows = min(AG_CHUNK, ncell - r0);
        mbar_wait(&sm->vbar[b], (uint32_t) ((c / AG_BUFS) & 1), &sm->aborted, P.abort_flag);
        for (int r = warp; r < nrows; r += AG_WARPS) {
            float vf[4], w[G];
            ag_row4(r0 + r == fresh ? sm->v_s : sm->vbuf[b][r], lane, vf);
#pragma unroll
            for (int i = 0; i < G; i += 2) *reinterpret_cast<float2 *>(w + i) = *reinterpret_cast<const float2 *>(S + (r0 + r) * G + i);
#pragma unroll
            for (int i = 0; i < G; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(vf[j], w[i], acc[i][j]);
        }
        if (c + AG_BUFS < nchunks) {
            __syncthreads();
            ag_issue(sm->vbuf[b], vc, EK, c + AG_BUFS, ncell, &sm->vbar[b]);
        }
    }
    __syncthreads();                                      // every copy into the buffers has landed and been read
    float * red = reinterpret_cast<float *>(sm->kbuf);
    static_assert(sizeof(float) * AG_WARPS * G * 128 <= sizeof(sm->kbuf) + sizeof(sm->vbuf), "partial sums");
#pragma unroll
    for (int i = 0; i < G; i++) *reinterpret_cast<float4 *>(red + (warp * G + i) * D + 4 * lane) = *reinterpret_cast<const float4 *>(acc[i]);
    __syncthreads();
    for (int i = tid; i < G * D; i += AG_THREADS) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < AG_WARPS; w++) t += red[w * G * D + i];
        (&sm->o_s[0][0])[i] = t;
    }
    if (splits > 1) ag_cluster_sync(); else __syncthreads();
    // two heads = one super-block of the q8_K activation (quantize_row_q8_K_ref, ggml-quants.c:3785-3822): a warp's work, dealt over the CTAs first
    const int sb = part + splits * warp;
    if (sb < G / 2) {
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = 0.f;
        for (int i = 0; i < splits; i++) {
            float y[8];
            ag_ld_f32x4(&sm->o_s[2 * sb][0] + 8 * lane, i, y);
            ag_ld_f32x4(&sm->o_s[2 * sb][0] + 8 * lane + 4, i, y + 4);
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] += y[j];
        }
        float4 * out = reinterpret_cast<float4 *>(P.out + (int64_t) (hk * G + 2 * sb) * D + 8 * lane);
        out[0] = make_float4(x[0], x[1], x[2], x[3]);
        out[1] = make_float4(x[4], x[5], x[6], x[7]);
        quantize_warp_q8K(x, lane, hk * (G / 2) + sb, P.outq);
    }
    if (splits > 1) ag_cluster_sync();                    // no CTA leaves while another may still read its part
}

template <int G> int launch_group(AgParams & P, int n_ctx, cudaStream_t stream, bool pdl) {
    // as many CTAs as a cluster may have and the machine holds, no more than there are chunks.  A step of four layers (32 heads over 8) in us, a CTA per head / a
    // cluster of 2 / 4 / 8: 1000 cells 320 / 304 / 274 / 260, 560 cells 284 / 284 / 263 / 260, 180 cells 250 / 260 / 250 / 251, 32 to 126 cells 246 .. 247 / 247 / 248 / 248 .. 250
    P.splits = AG_MAX_SPLIT;
    while (P.splits > 1 && (P.splits * P.n_head_kv > sm_count() || n_ctx <= AG_CHUNK * P.splits)) P.splits /= 2;
    const size_t smem = sizeof(AgSmem<G>) + (size_t) ((n_ctx + P.splits - 1) / P.splits) * G * sizeof(float);
    if (smem > 200 * 1024) return (int) cudaErrorNotSupported;
    static FuncAttrCache attr_cache;
    const cudaError_t e = ensure_dyn_smem(attr_cache, (const void *) k_attn_group<G>, smem, false);
    if (e != cudaSuccess) return (int) e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned) (P.n_head_kv * P.splits));
    cfg.blockDim = dim3(AG_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned) P.splits; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return (int) cudaLaunchKernelEx(&cfg, k_attn_group<G>, P);
}

}  // namespace

int launch_attn_group(const float * q, const float * k, const float * v, __half * kcache, __half * vcache, float * out, const ActQ & outq, int n_head, int n_head_kv, int D,
                      const int32_t * pos_dev, int n_ctx, const RopeParams & rp, const float * freq_factors, float scale, cudaStream_t stream, bool pdl) {
    if (D != 128 || n_head_kv <= 0 || n_head % n_head_kv || !outq.qs) return (int) cudaErrorNotSupported;
    AgParams P{q, k, v, kcache, vcache, out, outq, n_head_kv, 1, pos_dev, rp, freq_factors, scale, abort_flag()};
    switch (n_head / n_head_kv) {
    case 2: return launch_group<2>(P, n_ctx, stream, pdl);
    case 4: return launch_group<4>(P, n_ctx, stream, pdl);
    case 8: return launch_group<8>(P, n_ctx, stream, pdl);
    }
    return (int) cudaErrorNotSupported;
}

}  // namespace pb
