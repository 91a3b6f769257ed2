// prima.cpp_b200/csrc/latent_decode.cu — attention of one token per entry over the latent cache in one kernel: the query folded through W_uk, the walk over the
// rows, and W_uv on the weighted sum of latents (semantics: layers.h; latent.cu has the three kernels that serve what does not fit here).
// Bound: the way to memory and back.  A cluster of eight CTAs takes two heads of an entry.  Four CTAs share a head's maps, a quarter of the latent's entries of
// W_uk and a quarter of the rows of W_uv each, in registers and on their way before the kernel in front has ended, as are the cache rows of earlier
// tokens (only the token's own row is written in this pass, by a kernel in front).  The folded queries go to all CTAs of the cluster, each of
// which walks an eighth of the rows in stages of 16: scores with a warp to two rows, weighted sums with a thread to four entries of a head.  The sums go to the
// four CTAs of their head, which join them and apply W_uv.  The cut of the rows follows the sequence's own length, the choice
// between this kernel and those three the number of sequences: the order of the fp32 sums may change with it.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <atomic>

#include "launch.h"
#include "latent.cuh"
#include "layers.h"
#include "mixers.cuh"
#include "rows.cuh"
#include "tc.cuh"

namespace pb {
namespace {

constexpr int LD_CTAS = 8, LD_WARPS = 8, LD_THREADS = 32 * LD_WARPS, LD_HEADS = 2, LD_OF_HEAD = LD_CTAS / LD_HEADS, LD_ROWS = 16, LD_STAGES = 2;
constexpr int LD_RANK = 512, LD_ROW = 640, LD_DIM = 128;   // most entries of a latent, of a cache row, of a head

struct LatentDecode {
    const float * q; int64_t ldq;
    const int32_t * slot, * off, * pos0;
    LatentParams p;
    const __nv_bfloat16 * wuk, * wuv;
    const float * freq, * cache;
    int64_t slot_stride;
    const float * sink, * gate; int64_t ldg;
    void * out;
};

__device__ __forceinline__ void send4(float4 v, const float * at, int cta) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr(smem_u32(at), (uint32_t) cta)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

template <typename OT>
__global__ void __launch_bounds__(LD_THREADS, 2) __cluster_dims__(LD_CTAS, 1, 1) k_latent_decode_group(const __grid_constant__ LatentDecode P) {
    extern __shared__ __align__(16) float stage[];             // LD_STAGES x LD_ROWS cache rows
    __shared__ __align__(16) float qa[LD_HEADS][LD_ROW];       // folded queries, scaled
    __shared__ __align__(16) float got[LD_CTAS][LD_RANK];      // this CTA's head: the CTAs' weighted sums
    __shared__ float gotm[LD_CTAS], gotl[LD_CTAS], S[2][LD_HEADS][LD_ROWS];
    __shared__ __align__(16) float red[LD_WARPS][128];
    __shared__ float qs[LD_DIM];
    const LatentParams & p = P.p;
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int rank = blockIdx.x, h0 = blockIdx.y * LD_HEADS, e = blockIdx.z, hj = rank / LD_OF_HEAD, pj = rank % LD_OF_HEAD, h = h0 + hj;
    const int D = p.dim, Dr = p.rot_dim, R = p.kv_rank, RW = R + Dr, DV = p.vdim, H = p.heads, quarter = R / LD_OF_HEAD, share = (DV + LD_OF_HEAD - 1) / LD_OF_HEAD;
    const bool live = h < H;
    pdl_trigger();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const int t = P.off[e], pos = P.pos0[e];
    const int used = min(pos + 1, p.cache_rows), per = (used + LD_CTAS - 1) / LD_CTAS, r_lo = min(used, rank * per), r_hi = min(used, r_lo + per), own = pos % p.cache_rows;
    const float * rows = P.cache + (int64_t) P.slot[e] * P.slot_stride;
    // cache rows r0 .. into a stage: every row but the token's own, or that one alone
    auto fetch = [&](int r0, int s, bool the_own) {
        for (int j = warp; j < LD_ROWS; j += LD_WARPS) {
            const int r = r0 + j;
            if (r >= r_hi || (r == own) != the_own) continue;
            for (int i = 4 * lane; i < RW; i += 128) cp_async16(stage + (s * LD_ROWS + j) * RW + i, rows + (int64_t) r * RW + i, true);
        }
    };
#pragma unroll
    for (int s = 0; s < LD_STAGES; s++) fetch(r_lo + s * LD_ROWS, s, false);
    // the head's maps: W_uk rows 16 warp + i, four entries of the quarter a lane; W_uv rows 4 warp + i of the share, entries 8 lane and 256 + 8 lane
    uint2 uk[16];
    uint4 uv[4][2];
    const int rk = pj * quarter + 4 * lane, d0 = 16 * warp, v0 = pj * share + 4 * warp, v_hi = min(DV, (pj + 1) * share);
#pragma unroll
    for (int i = 0; i < 16; i++)
        uk[i] = live && 4 * lane < quarter && d0 + i < D ? *reinterpret_cast<const uint2 *>(P.wuk + ((int64_t) h * D + d0 + i) * R + rk) : make_uint2(0u, 0u);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < 2; c++)
            uv[i][c] = live && v0 + i < v_hi && 256 * c + 8 * lane < R ? *reinterpret_cast<const uint4 *>(P.wuv + ((int64_t) h * DV + v0 + i) * R + 256 * c + 8 * lane) : make_uint4(0u, 0u, 0u, 0u);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < LD_STAGES; s++) fetch(r_lo + s * LD_ROWS, s, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float * qr = P.q + (int64_t) t * P.ldq + (int64_t) h * (D + Dr);
    // the rotated part, by the first CTA of the head: a pair per thread, or an entry that does not turn
    const int half = p.rot_dims / 2;
    int ra = -1, rb = -1;
    float xa = 0.f, xb = 0.f;
    if (live && pj == 0 && tid < half) {
        pair_at(p, tid, ra, rb);
        turn(qr[D + ra], qr[D + rb], pos, P.freq[tid], p.rot_mag, xa, xb);
    } else if (live && pj == 0 && tid >= 2 * half && tid < Dr) {
        ra = tid;
        xa = qr[D + tid];
    } else if (!live && pj == 0 && tid < Dr) ra = tid;       // a head that is not there: zeros
    if (tid < D) qs[tid] = live ? qr[tid] : 0.f;
    __syncthreads();
    {
        float f[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float x = d0 + i < D ? qs[d0 + i] : 0.f;
            f[0] = fmaf(bf_lo(uk[i].x), x, f[0]); f[1] = fmaf(bf_hi(uk[i].x), x, f[1]);
            f[2] = fmaf(bf_lo(uk[i].y), x, f[2]); f[3] = fmaf(bf_hi(uk[i].y), x, f[3]);
        }
        *reinterpret_cast<float4 *>(&red[warp][4 * lane]) = make_float4(f[0], f[1], f[2], f[3]);
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every CTA of the cluster runs
    if (tid < quarter) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < LD_WARPS; w++) v += red[w][tid];
        v *= p.scale;
#pragma unroll
        for (int c = 0; c < LD_CTAS; c++) send(v, &qa[hj][pj * quarter + tid], c);
    }
    for (int c = 0; c < LD_CTAS; c++) {
        if (ra >= 0) send(xa * p.scale, &qa[hj][R + ra], c);
        if (rb >= 0) send(xb * p.scale, &qa[hj][R + rb], c);
    }
    cluster_barrier();
    constexpr int NC = LD_ROW / 128;
    float4 q[LD_HEADS][NC];
#pragma unroll
    for (int n = 0; n < LD_HEADS; n++)
#pragma unroll
        for (int c = 0; c < NC; c++) q[n][c] = 128 * c + 4 * lane < RW ? *reinterpret_cast<const float4 *>(&qa[n][128 * c + 4 * lane]) : make_float4(0.f, 0.f, 0.f, 0.f);
    // the walk: a stage's scores, then the weighted sums of head `vh`, entries 4 vr ..; every thread keeps its head's maximum and sum
    const int vh = tid >> 7, vr = 4 * (tid & 127);
    float m = -INFINITY, l = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    for (int r0 = r_lo, it = 0; r0 < r_hi; r0 += LD_ROWS, it++) {
        const int s = it & 1, nr = min(LD_ROWS, r_hi - r0);
        const float * tile = stage + s * LD_ROWS * RW;
        if (it >= LD_STAGES) asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                        // the stage is there, and the one before has been read
        if (it > 0) {
            fetch(r0 + LD_ROWS, s ^ 1, false);
            fetch(r0 + LD_ROWS, s ^ 1, true);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        {
            float v[4] = {0.f, 0.f, 0.f, 0.f};                  // head n, row warp + 8 j at 2 n + j
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int i = warp + LD_WARPS * j;
                    const float4 k = i < nr && 128 * c + 4 * lane < RW ? *reinterpret_cast<const float4 *>(tile + i * RW + 128 * c + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int n = 0; n < LD_HEADS; n++) v[2 * n + j] = fmaf(q[n][c].w, k.w, fmaf(q[n][c].z, k.z, fmaf(q[n][c].y, k.y, fmaf(q[n][c].x, k.x, v[2 * n + j]))));
                }
            joint_sum<4, 16>(v, lane);
            float x = v[0];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            const int i = warp + LD_WARPS * ((lane >> 3) & 1);
            if ((lane & 7) == 0) S[it & 1][lane >> 4][i] = i < nr ? x : -INFINITY;
        }
        __syncthreads();
        const float x = S[it & 1][vh][lane & 15];               // lanes 0 .. 15 and 16 .. 31 hold the same
        float mx = x;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float mn = fmaxf(m, mx), c = m == -INFINITY ? 0.f : expf(m - mn), w = x == -INFINITY ? 0.f : expf(x - mn);
        float sum = w;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        l = l * c + sum;
        acc = make_float4(acc.x * c, acc.y * c, acc.z * c, acc.w * c);
#pragma unroll
        for (int i = 0; i < LD_ROWS; i++) {
            const float wi = __shfl_sync(0xffffffffu, w, i);
            const float4 k = i < nr && vr < R ? *reinterpret_cast<const float4 *>(tile + i * RW + vr) : make_float4(0.f, 0.f, 0.f, 0.f);
            acc = make_float4(fmaf(wi, k.x, acc.x), fmaf(wi, k.y, acc.y), fmaf(wi, k.z, acc.z), fmaf(wi, k.w, acc.w));
        }
        m = mn;
    }
#pragma unroll
    for (int c = 0; c < LD_OF_HEAD; c++) {
        if (vr < R) send4(acc, &got[rank][vr], vh * LD_OF_HEAD + c);
        if (vr == 0) { send(m, &gotm[rank], vh * LD_OF_HEAD + c); send(l, &gotl[rank], vh * LD_OF_HEAD + c); }
    }
    cluster_barrier();
    if (!live) return;
    float M = -INFINITY, L = 0.f;
#pragma unroll
    for (int c = 0; c < LD_CTAS; c++) M = fmaxf(M, gotm[c]);
    float f[LD_CTAS];
#pragma unroll
    for (int c = 0; c < LD_CTAS; c++) {
        f[c] = gotm[c] == -INFINITY ? 0.f : expf(gotm[c] - M);
        L = fmaf(gotl[c], f[c], L);
    }
    if (P.sink && M != -INFINITY) L += expf(P.sink[h] - M);   // one more key in the denominator that has no value
    const float inv = L > 0.f ? 1.f / L : 0.f;
    // the joined latent entries of this lane, then four rows of W_uv
    float o[2][8];
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
        for (int i = 0; i < 8; i += 4) {
            const int r = 256 * c + 8 * lane + i;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < R)
#pragma unroll
                for (int n = 0; n < LD_CTAS; n++)
                    if (f[n] != 0.f) {
                        const float4 g = *reinterpret_cast<const float4 *>(&got[n][r]);
                        v = make_float4(fmaf(f[n], g.x, v.x), fmaf(f[n], g.y, v.y), fmaf(f[n], g.z, v.z), fmaf(f[n], g.w, v.w));
                    }
            o[c][i] = v.x * inv; o[c][i + 1] = v.y * inv; o[c][i + 2] = v.z * inv; o[c][i + 3] = v.w * inv;
        }
    float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const uint32_t u[4] = {uv[i][c].x, uv[i][c].y, uv[i][c].z, uv[i][c].w};
#pragma unroll
            for (int k = 0; k < 4; k++) y[i] = fmaf(bf_hi(u[k]), o[c][2 * k + 1], fmaf(bf_lo(u[k]), o[c][2 * k], y[i]));
        }
    joint_sum<4, 16>(y, lane);
    float x = y[0];
#pragma unroll
    for (int i = 4; i > 0; i >>= 1) x += __shfl_xor_sync(0xffffffffu, x, i);
    const int dv = v0 + (lane >> 3);
    if ((lane & 7) == 0 && dv < v_hi) put((OT *) P.out, (int64_t) t * H * DV + h * DV + dv, x * latent_gate(p, P.gate, (int64_t) t * P.ldg, h, dv));
}

}  // namespace

int launch_latent_decode_group(const float * q, int64_t ldq, const BatchView & b, const void * wuk, const void * wuv, int wtype, const LatentParams & p, const float * freq,
                               const float * cache, int64_t slot_stride, const float * sink, const float * gate, int64_t ldg, void * out, cudaStream_t st) {
    // A layer's step, us, three kernels / this, behind 8, 130 and 1024 rows: 16 heads, one sequence 49.8, 49.6, 59.0 / 37.8, 40.1, 50.5; four 72.8, 75.6, 93.5 / 66.5, 69.7,
    // 88.3; eight 81.0, 87.5, 106 / 65.0, 68.6, 96.1; 32 (256 clusters) 144, 149, 194 / 167, 185, 243.  8 heads, 32 sequences (128 clusters) 114, 127, 162 / 120,
    // 129, 163: with more clusters than the SMs hold at once the other way, which reads a row once for 16 heads, is ahead.
    if ((int64_t) b.n_entries * ((p.heads + LD_HEADS - 1) / LD_HEADS) > 96) return (int) cudaErrorNotSupported;
    if (wtype != T_BF16 || p.kv_rank > LD_RANK || p.kv_rank % 16 || p.dim > LD_DIM || p.vdim > LD_DIM || p.rot_dim % 4 || p.kv_rank + p.rot_dim > LD_ROW || p.rot_dim > LD_THREADS ||
        slot_stride % 4 || !at16(cache) || !at16(wuk) || !at16(wuv) || b.n_entries > 65535)
        return (int) cudaErrorNotSupported;
    const LatentDecode P{q, ldq, b.slot, b.off, b.pos0, p, (const __nv_bfloat16 *) wuk, (const __nv_bfloat16 *) wuv, freq, cache, slot_stride, sink, gate, ldg, out};
    const size_t smem = (size_t) LD_STAGES * LD_ROWS * (p.kv_rank + p.rot_dim) * sizeof(float);
    static FuncAttrCache cache_attr;
    const cudaError_t e = ensure_dyn_smem(cache_attr, (const void *) k_latent_decode_group<__nv_bfloat16>, smem, true);
    if (e != cudaSuccess) return (int) e;
    const dim3 grid(LD_CTAS, (unsigned) ((p.heads + LD_HEADS - 1) / LD_HEADS), (unsigned) b.n_entries);
    return ck_launch([&] { launch_dep(k_latent_decode_group<__nv_bfloat16>, grid, dim3(LD_THREADS), smem, st, P); });
}

}  // namespace pb
