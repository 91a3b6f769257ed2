// prima.cpp_b200/csrc/attn_group.cu — decode attention of the engine's per-token path over the f16 cache (row-major K and V, cell == position): rope(q),
// rope(k), cache store, softmax and the quantized activation of the output product in one launch.  The arithmetic is k_attn2's (ops.cu: FA-off
// numerics of the CPU backend, f16-rounded q and probabilities, fp32 sums); the work is laid out for contexts of more than a few cells.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "launch.h"
#include "quantize.cuh"
#include "rope.cuh"

namespace pb {
namespace {

// Two layouts, by the cells there are.
// Long contexts: one cluster per kv head, whose CTAs share the cells in equal consecutive parts; each serves all G query heads of the group, so that a cell is read
// once (one CTA per query head reads it G times and walks all of it alone: 24 us a launch at 1000 cells, 32 heads over 8; this 7).  The parts agree on each head's
// largest score and sum through distributed shared memory, CTA r adds super-block r of the group's output in the parts' order and quantizes it.
// Short ones (ag_head): a CTA per query head over all cells, nothing exchanged but results; what the other layout costs beside the cells (three cluster barriers, 64 KB of
// partial sums for a group of eight) is 3 us a layer there.
// Copies are counted by each thread's groups and a barrier of the CTA: an mbarrier on which 512 threads arrive cost 0.25 us a buffer and layer.
// Bound: a chain of small steps (load, rope, scores, exchanges, values, join).
// Buffers of 64 cells twice for K and V (twice of that cost a short context 6 us a layer).  Groups of two in 64 registers, so that two CTAs share an SM (a step of four layers
// at one cell 143 -> 139 us); groups of four and eight in 128 (2000 cells 276 -> 266 us).
// us of a step of four layers, a CTA per query head with all cells on their way (k_attn2, ops.cu) / this:
//   cells           1             32            128           180           256           257           400           1000          2000
//   32 heads / 8    229.5 / 229.6 230.6 / 228.5 236.8 / 233.6 241.6 / 237.3 245.0 / 241.1 248.2 / 243.8 258.2 / 245.0 305.2 / 251.0 385.2 / 266.1
//   64 heads / 8    519.3 / 520.8 520.1 / 523.1 526.4 / 526.4 531.0 / 530.6 534.5 / 532.9 537.7 / 538.1 547.9 / 539.5 594.9 / 549.1 675.7 / 570.0
//   16 heads / 8    139.1 / 138.1 140.1 / 137.5 143.8 / 140.0 148.6 / 143.8 152.1 / 147.2 155.8 / 155.0 166.0 / 155.6 212.7 / 161.6
//   32 heads / 4    228.0 / 230.2 229.3 / 228.1 235.0 / 232.6 239.8 / 236.7 243.1 / 240.3 246.2 / 248.4 256.3 / 249.9 303.2 / 258.8
constexpr int AG_THREADS = 512, AG_WARPS = 16, AG_CHUNK = 64, AG_BUFS = 2, AG_MAX_SPLIT = 8;
// Contexts of up to so many cells take a CTA per head: the chunks of keys that the four buffers hold.  The last ones are faster that way for every group (the table's 256
// and 257; a group of eight would be up to 290, by 1 %).
constexpr int AG_ALONE = 2 * AG_BUFS * AG_CHUNK;

template <int G> struct __align__(128) AgSmem {   // behind it: scores [cell of the part][G]
    __align__(128) __half kbuf[AG_BUFS][AG_CHUNK][128];
    __align__(128) __half vbuf[AG_BUFS][AG_CHUNK][128];   // both buffers, read out, take the warps' partial sums [AG_WARPS][G][128]
    uint64_t pair;                 // ag_head: the neighbour's result has arrived in o_s[1]
    volatile int aborted;          // wait watchdog (common.cuh)
    double x_sum[G];               // what the cluster's other CTAs read: this part's sums of exponentials, largest scores and weighed values
    float x_max[G];
    __align__(16) float o_s[G][128];
    double s_redd[AG_WARPS];
    float s_red[AG_WARPS];
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
// cells [c * AG_CHUNK, ...) of a part that starts at `cache`, if it has such: a group of this thread's copies either way
__device__ __forceinline__ void ag_issue(__half (*dst)[128], const __half * cache, int64_t row, int c, int ncell) {
    const int r0 = c * AG_CHUNK, pieces = min(AG_CHUNK, ncell - r0) * 16;
    for (int i = threadIdx.x; i < pieces; i += AG_THREADS) {
        const int r = i >> 4, p = i & 15;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&dst[r][p * 8])), "l"(cache + (int64_t) (r0 + r) * row + p * 8) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// all threads' copies have landed but for the last `after` groups of each
template <int after> __device__ __forceinline__ void ag_landed() {
    asm volatile("cp.async.wait_group %0;" ::"n"(after) : "memory");
    __syncthreads();
}
__device__ __forceinline__ void ag_row4(const __half * row, int lane, float (&f)[4]) {
    const uint2 raw = *reinterpret_cast<const uint2 *>(row + 4 * lane);
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&raw.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&raw.y));
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}

// A short context: CTA h takes query head h over all cells.  Pairs of heads lie in one cluster; the odd one's result goes into the even one's shared memory, which quantizes
// their super-block.  Keys of up to four chunks travel ahead of the wait, in all the buffers; values of more than two follow chunk by chunk behind the scores.
// The first CTAs of the grid take the heads, whatever cluster they are in: with the group's own cluster, half of each idle, a layer cost 0.5 us more.
template <int G>
__device__ __forceinline__ void ag_head(const AgParams & P, AgSmem<G> * sm, float * S, int h, int pos) {
    constexpr int D = 128;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hk = h / G, even_rank = h % P.splits & ~1, ncell = pos + 1, nchunks = (ncell + AG_CHUNK - 1) / AG_CHUNK;
    const int64_t EK = (int64_t) P.n_head_kv * D;
    const __half * kc = P.kc + hk * D, * vc = P.vc + hk * D;
    if (tid == 0) {
        mbar_init(&sm->pair, 1);
        sm->aborted = 0;
        mbar_fence_init();
        if ((h & 1) == 0) mbar_arrive_expect_tx(&sm->pair, D * 4);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // the even CTA is there; the odd one looks before it writes
    auto buf = [&](int i) { return i < AG_BUFS ? sm->kbuf[i] : sm->vbuf[i - AG_BUFS]; };
    const int v0 = nchunks <= AG_BUFS ? AG_BUFS : 0;      // value chunk c lies in buffer v0 + c
    for (int c = 0; c < nchunks; c++) ag_issue(buf(c), kc, EK, c, ncell);
    if (v0)
        for (int c = 0; c < AG_BUFS; c++) ag_issue(buf(v0 + c), vc, EK, c, ncell);
    const RopeParams & rp = P.rp;
    const int half_dims = rp.n_dims / 2;
    const bool neox = rp.mode & 2;
    if (tid < 64 && tid < half_dims) {
        float c, s;
        rope_cos_sin(rp, pos, tid, P.freq_factors, c, s);
        sm->cs[tid][0] = c; sm->cs[tid][1] = s;
    }
    pdl_wait();
    const int pair = tid & 63, i0 = neox ? pair : 2 * pair, i1 = neox ? pair + half_dims : 2 * pair + 1;
    const float * src = tid < 64 ? P.q + (int64_t) h * D : tid < 128 ? P.k + (int64_t) hk * D : P.v + (int64_t) hk * D;
    float x0 = 0.f, x1 = 0.f;
    if (tid < 128) {
        if (pair < half_dims) { x0 = __ldcg(src + i0); x1 = __ldcg(src + i1); }
    } else if (tid < 256) x0 = __ldcg(src + tid - 128);
    __syncthreads();                                      // the angles
    if (tid < 128) {
        auto keep = [&](int j, float y) {
            const __half v = __float2half_rn(y);
            if (tid < 64) sm->q_s[0][j] = __half2float(v);
            else sm->k_s[j] = v;
        };
        if (pair < half_dims) {
            float y0, y1;
            rope_rotate(x0, x1, sm->cs[pair][0], sm->cs[pair][1], y0, y1);
            keep(i0, y0);
            keep(i1, y1);
        }
        for (int j = rp.n_dims + pair; j < D; j += 64) keep(j, __ldcg(src + j));
    } else if (tid < 256) sm->v_s[tid - 128] = __float2half_rn(x0);
    if (v0) ag_landed<AG_BUFS>(); else ag_landed<0>();    // the keys
    if (h % G == 0 && warp == 0) {
        const int64_t at = (int64_t) pos * EK + hk * D + 4 * lane;
        *reinterpret_cast<uint2 *>(P.kc + at) = *reinterpret_cast<const uint2 *>(sm->k_s + 4 * lane);
        *reinterpret_cast<uint2 *>(P.vc + at) = *reinterpret_cast<const uint2 *>(sm->v_s + 4 * lane);
    }
    float q[4];
    *reinterpret_cast<float4 *>(q) = *reinterpret_cast<const float4 *>(&sm->q_s[0][4 * lane]);
    for (int c = 0; c < nchunks; c++) {
        const int p0 = c * AG_CHUNK, nrows = min(AG_CHUNK, ncell - p0);
        float v[AG_CHUNK / AG_WARPS];                     // a warp's four cells of the chunk, summed over the lanes together (the order of a sum is that of warp_sum)
#pragma unroll
        for (int k = 0; k < AG_CHUNK / AG_WARPS; k++) {
            const int i = warp + AG_WARPS * k;
            float kf[4];
            ag_row4(p0 + i == pos ? sm->k_s : buf(c)[i], lane, kf);
            v[k] = fmaf(kf[3], q[3], fmaf(kf[2], q[2], fmaf(kf[1], q[1], kf[0] * q[0])));
        }
        static_assert(AG_CHUNK / AG_WARPS == 4, "cells of a warp");
        const bool hi = lane & 16, odd = lane & 8;
#pragma unroll
        for (int k = 0; k < 2; k++) v[k] = (hi ? v[k + 2] : v[k]) + __shfl_xor_sync(0xffffffffu, hi ? v[k] : v[k + 2], 16);
        v[0] = (odd ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[1], 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        const int i = warp + AG_WARPS * (lane >> 3);      // hi: cells 2 and 3, odd: 1 and 3
        if ((lane & 7) == 0 && i < nrows) S[p0 + i] = __fmul_rn(v[0], P.scale);
        if (!v0) {                                        // every warp is done with the chunk: its values take the place
            __syncthreads();
            ag_issue(buf(c), vc, EK, c, ncell);
        }
    }
    if (v0) ag_landed<0>();                               // the values, and every warp's scores
    // every warp takes the softmax's maximum and sum for itself: no barrier
    float m = -INFINITY, e[AG_ALONE / 32];
#pragma unroll
    for (int i = 0; i < AG_ALONE / 32; i++) {
        e[i] = 32 * i + lane < ncell ? S[32 * i + lane] : -INFINITY;
        m = fmaxf(m, e[i]);
    }
    m = warp_max(m);
    double sum = 0.0;
#pragma unroll
    for (int i = 0; i < AG_ALONE / 32; i++) {
        if (32 * i >= ncell) break;
        e[i] = 32 * i + lane < ncell ? expf(__fsub_rn(e[i], m)) : 0.f;
        sum += (double) e[i];
    }
    sum = warp_sum_d(sum);
    const float inv = (float) (1.0 / sum);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (!v0) ag_landed<0>();
#pragma unroll
    for (int c = 0; c < 2 * AG_BUFS; c++) {
        if (c >= nchunks) break;
        const int p0 = c * AG_CHUNK, nrows = min(AG_CHUNK, ncell - p0);
#pragma unroll
        for (int k = 0; k < AG_CHUNK / AG_WARPS; k++) {   // cell p0 + i: lane i % 32 of this chunk's weights has it
            const int i = warp + AG_WARPS * k;
            const float w = __half2float(__float2half_rn(__fmul_rn(__shfl_sync(0xffffffffu, e[c * (AG_CHUNK / 32) + (AG_WARPS * k) / 32], i & 31), inv)));
            if (i >= nrows) continue;
            float vf[4];
            ag_row4(p0 + i == pos ? sm->v_s : buf(v0 + c)[i], lane, vf);
#pragma unroll
            for (int j = 0; j < 4; j++) acc[j] = fmaf(vf[j], w, acc[j]);
        }
    }
    __syncthreads();                                      // every copy has landed and been read: the buffers take the warps' sums
    float * red = reinterpret_cast<float *>(sm->kbuf);
    *reinterpret_cast<float4 *>(red + warp * D + 4 * lane) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __syncthreads();
    if (tid < D) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < AG_WARPS; w++) t += red[w * D + tid];
        P.out[(int64_t) h * D + tid] = t;
        if ((h & 1) == 0) sm->o_s[0][tid] = t;
        else asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(ag_remote(&sm->o_s[1][tid], even_rank)), "r"(__float_as_uint(t)), "r"(ag_remote(&sm->pair, even_rank)) : "memory");
    }
    if (h & 1) return;
    __syncthreads();
    if (warp == 0) {
        mbar_wait(&sm->pair, 0u, &sm->aborted, P.abort_flag);
        float x[8];                                       // lanes 0 .. 15: this head's entries, 16 .. 31: the next one's
        const float * o = &sm->o_s[0][0] + 8 * lane;
        *reinterpret_cast<float4 *>(x) = *reinterpret_cast<const float4 *>(o);
        *reinterpret_cast<float4 *>(x + 4) = *reinterpret_cast<const float4 *>(o + 4);
        quantize_warp_q8K(x, lane, h / 2, P.outq);
    }
}

template <int G>
__global__ void __launch_bounds__(AG_THREADS, G == 2 ? 2 : 1) k_attn_group(const __grid_constant__ AgParams P) {
    constexpr int D = 128;
    extern __shared__ __align__(128) uint8_t ag_raw[];
    AgSmem<G> * sm = reinterpret_cast<AgSmem<G> *>(ag_raw);
    float * S = reinterpret_cast<float *>(ag_raw + sizeof(AgSmem<G>));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int part = blockIdx.x % P.splits, hk = blockIdx.x / P.splits;
    const int64_t EK = (int64_t) P.n_head_kv * D;
    pdl_trigger();
    // ---- independent of the product in front: the position (written before this token's first kernel), cache cells of earlier tokens
    const int pos = *P.pos_dev, all = pos + 1;
    if (all <= AG_ALONE) {   // the first CTAs take a head each, pairs of heads in one cluster; the others leave (exited threads take no part in a cluster's barriers)
        if ((int) blockIdx.x < P.n_head_kv * G) ag_head<G>(P, sm, S, blockIdx.x, pos);
        return;
    }
    const int splits = P.splits;
    const int per = (all + splits - 1) / splits, cell0 = min(part * per, all), ncell = min(per, all - cell0);   // the last parts may have no cell
    const int fresh = pos - cell0;                        // this token's cell, taken from shared memory; < ncell in the last part that has cells only
    const int nchunks = (ncell + AG_CHUNK - 1) / AG_CHUNK;
    const __half * kc = P.kc + (int64_t) cell0 * EK + hk * D, * vc = P.vc + (int64_t) cell0 * EK + hk * D;
#pragma unroll
    for (int c = 0; c < AG_BUFS; c++) ag_issue(sm->kbuf[c], kc, EK, c, ncell);
#pragma unroll
    for (int c = 0; c < AG_BUFS; c++) ag_issue(sm->vbuf[c], vc, EK, c, ncell);
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
        if (c < AG_BUFS) ag_landed<2 * AG_BUFS - 1>(); else ag_landed<AG_BUFS - 1>();
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
        if (c + AG_BUFS < nchunks) __syncthreads();       // every warp is done with this buffer
        ag_issue(sm->kbuf[b], kc, EK, c + AG_BUFS, ncell);
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
    ag_cluster_sync();
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
    ag_cluster_sync();
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
        if (c == 0) ag_landed<0>(); else if (c >= AG_BUFS) ag_landed<AG_BUFS - 1>();
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
        if (c + AG_BUFS < nchunks) __syncthreads();
        ag_issue(sm->vbuf[b], vc, EK, c + AG_BUFS, ncell);
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
    ag_cluster_sync();
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
    ag_cluster_sync();                    // no CTA leaves while another may still read its part
}

template <int G> int launch_group(AgParams & P, int n_ctx, cudaStream_t stream, bool pdl) {
    // as many CTAs as a cluster may have and the machine holds, no more than there are chunks, but one for every head of the group.  A step of four layers (32 heads over
    // 8) in us by the cells' parts, 2 / 4 / 8: 1000 cells 304 / 274 / 260, 560 cells 284 / 263 / 260 (taken while a buffer had a barrier of 512 arrivals)
    P.splits = AG_MAX_SPLIT;
    while (P.splits > G && (P.splits * P.n_head_kv > sm_count() || n_ctx <= AG_CHUNK * P.splits)) P.splits /= 2;
    const size_t smem = sizeof(AgSmem<G>) + std::max<size_t>((size_t) ((n_ctx + P.splits - 1) / P.splits) * G, AG_ALONE) * sizeof(float);
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
