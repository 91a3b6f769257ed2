// prima.cpp_b200/csrc/dense_stream.cu — bf16 dense product for up to four tokens, weights streamed through shared memory:
//   C[t][n] = alpha * sum_k A[t][k] W[n][k] (+ bias[n]) (+ resid[t][n])   or the gated unit of row pairs (DenseAct::silu_glu),
// where A is given, or is the RMS norm of fp32 rows (every CTA makes it for itself: one kernel and its way through L2 less in front of a product).
// Bound: the weights' way from HBM, and for a few MB the start and end of a kernel.  One CTA per SM takes an equal share of the rows, which lie one
// behind the other in memory.  Each of its 16 warps brings pieces of 4 KB by bulk copies into a ring of its own, two pieces deep, so that 128 KB
// are on their way whatever the registers hold; the ring fills before the kernel in front has ended (weights depend on nothing).  A CTA asks for more than
// half of an SM's shared memory: two of one launch on one SM would finish last.  A piece is in registers, and its successor asked for, before it is multiplied.
// The pieces' sums of a row meet in their order at the end.
// A token of a six-layer model of width 2048 (generate, one request): 435 us with a warp to a row and norms of their own, 397 with this.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "launch.h"
#include "layers.h"
#include "mixers.cuh"

namespace pb {
namespace {

constexpr int ST_WARPS = 16, ST_THREADS = ST_WARPS * 32, ST_SLOTS = 2, ST_PIECE = 4096, ST_PARTS = 2048, ST_NORM_V = 4;

struct StreamParams {
    const __nv_bfloat16 * A; int64_t lda;
    const float * x; const int32_t * rows; const float * nw; float eps;   // instead of A: K numbers of row t, or rows[t] (lda apart), to be normed; the norm's weight
    const __nv_bfloat16 * W;
    float * C; int64_t ldc;
    const float * bias; const float * resid; int64_t ldr;
    float alpha;
    int T, N, K;          // N: results of a token (pairs of rows with a gated unit)
    int segs;             // pieces of a row
    int * abort_flag;
    DenseAct act;
};
struct StreamCtl {
    uint64_t full[ST_WARPS][ST_SLOTS];
    float red[33];
    int abort;
};

__device__ __forceinline__ void unpack8(const uint4 & v, float (&f)[8]) {
    const uint32_t r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) { f[2 * i] = __uint_as_float(r[i] << 16); f[2 * i + 1] = __uint_as_float(r[i] & 0xffff0000u); }
}

// TB: tokens; RB rows x SEG entries make a piece; NORM: A is made here
template <int TB, int RB, bool NORM>
__global__ void __launch_bounds__(ST_THREADS, 1) k_dense_stream(const __grid_constant__ StreamParams P) {
    constexpr int SEG = ST_PIECE / 2 / RB, NC = SEG / 256;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float parts[ST_PARTS];                 // [row][piece][token]
    __shared__ StreamCtl ctl;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int R = P.act.silu_glu ? 2 : 1;
    pdl_trigger();
    // rows of this CTA: the first N % CTAs of them take one result more
    const int each = P.N / (int) gridDim.x, more = P.N - each * (int) gridDim.x, u_lo = each * (int) blockIdx.x + min((int) blockIdx.x, more);
    const int nrows = R * (each + ((int) blockIdx.x < more ? 1 : 0));
    uint8_t * ring = smem + warp * (ST_SLOTS * ST_PIECE), * abase = smem + ST_WARPS * ST_SLOTS * ST_PIECE;   // then A [token][segs * SEG]
    const uint8_t * src = reinterpret_cast<const uint8_t *>(P.W) + (int64_t) R * u_lo * P.K * 2;
    const uint64_t policy = policy_evict_first();
    // a warp's place in the row of pieces: every ST_WARPS-th one is its own
    const int per = ST_WARPS / P.segs, dr = per * RB, dg = ST_WARPS - per * P.segs, first = warp / P.segs;
    struct Place { int r, g, slot; uint32_t phase; };
    auto next = [&](Place & p) {
        p.r += dr; p.g += dg;
        if (p.g >= P.segs) { p.g -= P.segs; p.r += RB; }
        if (++p.slot == ST_SLOTS) { p.slot = 0; p.phase ^= 1u; }
    };
    Place in{first * RB, warp - first * P.segs, 0, 0u}, at = in;
    auto fetch = [&]() {                              // one lane
        const int k0 = in.g * SEG, nr = min(RB, nrows - in.r);
        const uint32_t bytes = 2u * (uint32_t) min(SEG, P.K - k0);
        mbar_arrive_expect_tx(&ctl.full[warp][in.slot], bytes * (uint32_t) nr);
#pragma unroll
        for (int i = 0; i < RB; i++)
            if (i < nr) bulk_g2s(ring + in.slot * ST_PIECE + i * (2 * SEG), src + ((int64_t) (in.r + i) * P.K + k0) * 2, bytes, &ctl.full[warp][in.slot], policy);
    };
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < ST_SLOTS; s++) mbar_init(&ctl.full[warp][s], 1);
        if (warp == 0) ctl.abort = 0;
        mbar_fence_init();
    }
#pragma unroll
    for (int s = 0; s < ST_SLOTS; s++) {
        if (in.r >= nrows) break;
        if (lane == 0) fetch();
        next(in);
    }
    const int apad = P.segs * SEG, keep = ST_PARTS / (TB * P.segs * RB) * RB & ~1;   // rows whose sums fit
    // one token: what a result meets arrives beside the weights (a product that makes its norm meets nothing)
    const bool early = !NORM && TB == 1 && R == 1 && nrows <= min(keep, ST_THREADS);
    float meet = 0.f;
    if constexpr (NORM) {
        float4 wn[ST_NORM_V];
#pragma unroll
        for (int i = 0; i < ST_NORM_V; i++) {
            const int k = 4 * (tid + i * ST_THREADS);
            wn[i] = k < P.K ? *reinterpret_cast<const float4 *>(P.nw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        pdl_wait();
        for (int t = 0; t < P.T; t++) {
            const float * xr = P.x + (int64_t) (P.rows ? P.rows[t] : t) * P.lda;
            float4 v[ST_NORM_V];
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < ST_NORM_V; i++) {
                const int k = 4 * (tid + i * ST_THREADS);
                v[i] = k < P.K ? *reinterpret_cast<const float4 *>(xr + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < ST_NORM_V; i++) s += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
            const float inv = 1.f / sqrtf(block_sum(s, ctl.red) / (float) P.K + P.eps);
#pragma unroll
            for (int i = 0; i < ST_NORM_V; i++) {
                const int k = 4 * (tid + i * ST_THREADS);
                if (k < P.K) {
                    __nv_bfloat162 * y = reinterpret_cast<__nv_bfloat162 *>(abase + 2 * (t * apad + k));
                    y[0] = __floats2bfloat162_rn(v[i].x * inv * wn[i].x, v[i].y * inv * wn[i].y);
                    y[1] = __floats2bfloat162_rn(v[i].z * inv * wn[i].z, v[i].w * inv * wn[i].w);
                }
            }
        }
        for (int i = tid; i < TB * apad; i += ST_THREADS) {   // entries past K, rows past T
            const int t = TB == 1 ? 0 : i / apad, k = i - t * apad;
            if (t >= P.T || k >= P.K) *reinterpret_cast<__nv_bfloat16 *>(abase + 2 * i) = __float2bfloat16_rn(0.f);
        }
    } else {
        pdl_wait();
        if (early && tid < nrows && P.resid) meet = P.resid[u_lo + tid];
        for (int i = tid * 8; i < TB * apad; i += ST_THREADS * 8) {
            const int t = TB == 1 ? 0 : i / apad, k = i - t * apad;
            *reinterpret_cast<uint4 *>(abase + 2 * i) = t < P.T && k < P.K ? *reinterpret_cast<const uint4 *>(P.A + (int64_t) t * P.lda + k) : make_uint4(0u, 0u, 0u, 0u);
        }
    }
    __syncthreads();
    int base = 0;                                     // rows whose results are written
    auto finish = [&](int done) {                     // results of rows [base, done)
        __syncthreads();
        const int nu = (done - base) / R, u0 = u_lo + base / R;
        for (int t = 0; t < P.T; t++)
            for (int u = tid; u < nu; u += ST_THREADS) {
                const int n = u0 + u;
                auto sum = [&](int row) {
                    const float * p = parts + row * P.segs * TB + t;
                    float v = 0.f;
                    for (int g = 0; g < P.segs; g++) v += p[g * TB];
                    return P.alpha * v;
                };
                if (R == 2) {
                    const float g = sum(2 * u), v = sum(2 * u + 1);
                    put((__nv_bfloat16 *) P.act.y, (int64_t) t * P.act.ldy + n, silu_f(g) * v);
                    continue;
                }
                float v = sum(u);
                if (P.bias) v += P.bias[n];
                if constexpr (!NORM) {
                    if (early) v += meet;
                    else if (P.resid) v += P.resid[(int64_t) t * P.ldr + n];
                }
                if (P.act.xielu) put((__nv_bfloat16 *) P.act.y, (int64_t) t * P.act.ldy + n, xielu_f(v, softplus_f(P.act.xielu[0]), 0.5f + softplus_f(P.act.xielu[1])));
                else P.C[(int64_t) t * P.ldc + n] = v;
            }
        base = done;
    };
    while (base < nrows) {
        const int top = min(nrows, base + keep);
        while (at.r < top) {
            mbar_wait(&ctl.full[warp][at.slot], at.phase, &ctl.abort, P.abort_flag);
            const int k0 = at.g * SEG, left = P.K - k0 - 8 * lane;
            const uint8_t * w8 = ring + at.slot * ST_PIECE + 16 * lane, * a8 = abase + 2 * k0 + 16 * lane;
            uint4 w[RB][NC];
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int i = 0; i < RB; i++) w[i][c] = c * 256 < left ? *reinterpret_cast<const uint4 *>(w8 + i * (2 * SEG) + c * 512) : make_uint4(0u, 0u, 0u, 0u);
            uint32_t some = 0u;
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int i = 0; i < RB; i++) some ^= w[i][c].x;
            loads_done(some);
            __syncwarp();
            if (in.r < nrows) {
                if (lane == 0) fetch();
                next(in);
            }
            float acc[2][RB * TB];
#pragma unroll
            for (int i = 0; i < RB * TB; i++) acc[0][i] = acc[1][i] = 0.f;
#pragma unroll
            for (int c = 0; c < NC; c++) {
#pragma unroll
                for (int t = 0; t < TB; t++) {
                    float a[8];
                    unpack8(*reinterpret_cast<const uint4 *>(a8 + t * 2 * apad + c * 512), a);
#pragma unroll
                    for (int i = 0; i < RB; i++) {
                        float b[8];
                        unpack8(w[i][c], b);
#pragma unroll
                        for (int q = 0; q < 8; q++) acc[c & 1][i * TB + t] = fmaf(a[q], b[q], acc[c & 1][i * TB + t]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < RB * TB; i++) acc[0][i] = wsum(acc[0][i] + acc[1][i]);
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < RB; i++)
#pragma unroll
                    for (int t = 0; t < TB; t++) parts[((at.r - base + i) * P.segs + at.g) * TB + t] = acc[0][i * TB + t];
            }
            next(at);
        }
        finish(top);
        if (top < nrows) __syncthreads();
    }
}

template <int TB, int RB, bool NORM>
int launch_stream(StreamParams P, cudaStream_t st) {
    constexpr int SEG = ST_PIECE / 2 / RB;
    P.segs = (P.K + SEG - 1) / SEG;
    const size_t smem = (size_t) ST_WARPS * ST_SLOTS * ST_PIECE + (size_t) TB * P.segs * SEG * 2;
    if (smem + sizeof(float) * ST_PARTS + sizeof(StreamCtl) > 226 * 1024) return (int) cudaErrorNotSupported;
    static FuncAttrCache cache;
    const cudaError_t e = ensure_dyn_smem(cache, (const void *) k_dense_stream<TB, RB, NORM>, smem, true);
    if (e != cudaSuccess) return (int) e;
    g_launches++;
    return launch_dep(k_dense_stream<TB, RB, NORM>, dim3((unsigned) std::min(sm_count(), P.N)), dim3(ST_THREADS), smem, st, P);
}

template <bool NORM>
int launch_tokens(const StreamParams & P, cudaStream_t st) {
    if (P.T == 1) return launch_stream<1, 1, NORM>(P, st);
    if (P.T == 2) return launch_stream<2, 1, NORM>(P, st);
    return launch_stream<4, 2, NORM>(P, st);
}

// Calls one by one from HBM, us, a warp to a row with its loads in registers (dense.cu) / this, for 1, 2 and 4 tokens: 2048 x 2048 6.3, 8.3, 8.7 / 6.3, 7.6,
// 8.3; 16384 x 2048 17.4, 21.1, 27.7 / 17.0, 19.0, 23.1; 2048 x 8192 10.9, 12.8, 14.8 / 11.6, 12.8, 16.4; 4096 x 14336 26.3, 31.8, - / 26.3, 28.3, -;
// 28672 x 4096 49.7, 53.1, 69.1 / 45.6, 41.1, 55.3; 1000 x 5504 8.3, 8.6, 12.4 / 8.3, 9.1, 10.4; 388 x 2048 6.2 / 5.1.  So three and four tokens of rows
// beyond 6144 entries, whose operands every CTA would stage for a few rows, stay there.
bool stream_ok(const __nv_bfloat16 * W, int64_t ldw, int T, int K) {
    return T >= 1 && T <= 4 && K >= 256 && K <= (T <= 2 ? 16384 : 6144) && K % 8 == 0 && ldw == K && ((uintptr_t) W & 15) == 0;
}

// A product by itself has no kernel in front beside whose end its rings could fill, which is what it gains in a pass (generate with ff 4096 to 8192, widths 1024 to 2048, one to four requests:
// 0 to 9 % of a call).  What is left are few rounds of pieces, where a launch counts, and many bytes.  The same times as above, 1 / 2 / 4 tokens, rows over this: 300 x 3072 1.46 / 1.34 / 1.59;
// 1000 x 3072 1.32 / 1.12 / 1.28; 2048 x 2048 0.99 / 1.09 / 1.04; 4096 x 2048 0.99 / 0.91 / 0.94; 2048 x 5504 0.90 / 0.84 / 0.88; 1000 x 11008 0.83 / 0.84; 8192 x 1024 (half of a piece) 0.83 / 0.80 / 0.99;
// 4096 x 4096 0.92 / 1.00 / 1.11; 8192 x 4096 1.02 / 1.04 / 1.21; 16384 x 4096 1.00 / 1.24 / 1.44.
bool alone_ok(int T, int N, int K) {
    const int seg = T <= 2 ? ST_PIECE / 2 : ST_PIECE / 4;
    return (int64_t) N * ((K + seg - 1) / seg * seg) <= (T <= 2 ? 5 << 20 : 6 << 20) || (K >= 2048 && (int64_t) N * K >= (T == 4 ? 16 << 20 : 32 << 20));
}

}  // namespace

int launch_dense_stream(const __nv_bfloat16 * A, int64_t lda, const __nv_bfloat16 * W, int64_t ldw, float * C, int64_t ldc, int T, int N, int K, const float * bias,
                        const float * resid, int64_t ldr, float alpha, cudaStream_t st, const DenseAct & act, bool alone) {
    if (!stream_ok(W, ldw, T, K) || (alone && !alone_ok(T, N, K)) || lda % 8 || ((uintptr_t) A & 15)) return (int) cudaErrorNotSupported;
    return launch_tokens<false>(StreamParams{A, lda, nullptr, nullptr, nullptr, 0.f, W, C, ldc, bias, resid, ldr, alpha, T, act.silu_glu ? N / 2 : N, K, 1, abort_flag(), act}, st);
}

int launch_dense_normed(int type, const float * x, int64_t ldx, const int32_t * rows, const float * norm_w, float eps, const void * W, int64_t ldw, float * C, int64_t ldc, int T, int N, int K,
                        const float * bias, cudaStream_t st, const DenseAct & act) {
    const __nv_bfloat16 * w = (const __nv_bfloat16 *) W;
    if (type != T_BF16 || !stream_ok(w, ldw, T, K) || K > 4 * ST_NORM_V * ST_THREADS || ldx % 4 || ((uintptr_t) x & 15) || ((uintptr_t) norm_w & 15) || N <= 0 || (act.silu_glu && N % 2))
        return (int) cudaErrorNotSupported;
    return launch_tokens<true>(StreamParams{nullptr, ldx, x, rows, norm_w, eps, w, C, ldc, bias, nullptr, 0, 1.f, T, act.silu_glu ? N / 2 : N, K, 1, abort_flag(), act}, st);
}

}  // namespace pb
