// prima.cpp_b200/csrc/attn_decode.cu — attention of one token per entry over the slot's cache, for the layer-list models: a cluster of eight CTAs per
// (entry, kv head).  Semantics (window, kept first tokens, chunks, soft-cap, sink, gate) as k_attn_window_decode in mixers.cu, which serves what does not fit here.
// Bound: the way to memory and back, a few times in a row.  Each CTA takes an eighth of the rows the sequence has so far, for all query heads of the
// kv head, so that a row is read once; it asks for the rows of earlier tokens before the kernel in front has ended (only the token's own row is
// written in this pass, by a kernel in front).  A stage of 32 rows: scores with a warp to a row, softmax with a warp to a head, weighted values with a warp
// to a head and a share of the rows.  The CTAs send their sums to the CTA that finishes an output entry: one cluster barrier and no second kernel.
// The cut of the rows follows the sequence's own length.  Which kernel takes a call follows the sequences beside it (launch_attn_decode_group below), and with it the order of the fp32 sums.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <atomic>

#include "attn.cuh"
#include "launch.h"
#include "layers.h"
#include "mixers.cuh"
#include "rows.cuh"
#include "tc.cuh"

namespace pb {
namespace {

constexpr int AD_CTAS = 8, AD_WARPS = 8, AD_ROWS = 32, AD_DIM = 128, AD_BYTES = 64 * 1024;

struct DecodeParams {
    AttnIO io;
    const int32_t * slot, * off, * pos0;
    AttnParams a;
    const float * kc, * vc;
    int64_t slot_stride;
    void * out;
};

// GM: query heads of a kv head (at most); TIED: a key is its own value
template <typename OT, int GM, bool TIED>
__global__ void __launch_bounds__(AD_WARPS * 32) __cluster_dims__(AD_CTAS, 1, 1) k_attn_decode_group(const __grid_constant__ DecodeParams P) {
    constexpr int PARTS = AD_WARPS / GM;                  // shares of a stage's rows in the value sums
    constexpr int TILE = AD_ROWS * AD_DIM * (TIED ? 1 : 2), SLICE = GM * AD_DIM / AD_CTAS, STAGES = AD_BYTES / (4 * TILE);
    extern __shared__ __align__(16) float stage[];        // stages of AD_ROWS keys [D], then AD_ROWS values [DV]
    __shared__ float S[GM][AD_ROWS], corr[GM], runm[GM], runl[GM];
    __shared__ __align__(16) float sums[PARTS][GM][AD_DIM];
    __shared__ float got[AD_CTAS][SLICE], gotm[AD_CTAS][GM], gotl[AD_CTAS][GM];
    const AttnParams & a = P.a;
    const int rank = blockIdx.x, kvh = blockIdx.y, e = blockIdx.z;
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int D = a.dim, DV = TIED ? D : a.vdim, G = a.heads / a.kv_heads;
    pdl_trigger();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const int t = P.off[e], pi = P.pos0[e];
    const int keep = min(a.keep_first, a.cache_rows), ring = a.cache_rows - keep;
    const int used = dec_rows_used(a, pi), per = (used + AD_CTAS - 1) / AD_CTAS, r_lo = min(used, rank * per), r_hi = min(used, r_lo + per);
    const int own = cache_row(pi, keep, max(ring, 1));
    const float * kc = P.kc + (int64_t) P.slot[e] * P.slot_stride + kvh * D, * vc = P.vc + (int64_t) P.slot[e] * P.slot_stride + kvh * DV;
    // rows [r0, r0 + AD_ROWS) of the share into a stage: every row but the token's own, or that one alone
    auto fetch = [&](int r0, int s, bool the_own) {
        for (int i = warp; i < AD_ROWS && r0 + i < r_hi; i += AD_WARPS) {
            if ((r0 + i == own) != the_own) continue;
            float * k = stage + s * TILE + i * AD_DIM;
            if (4 * lane < D) cp_async16(k + 4 * lane, kc + (int64_t) (r0 + i) * P.io.k_row + 4 * lane, true);
            if (!TIED && 4 * lane < DV) cp_async16(k + AD_ROWS * AD_DIM + 4 * lane, vc + (int64_t) (r0 + i) * P.io.v_row + 4 * lane, true);
        }
    };
#pragma unroll
    for (int s = 0; s < STAGES; s++) fetch(r_lo + s * AD_ROWS, s, false);
    if (tid < GM) { runm[tid] = -INFINITY; runl[tid] = 0.f; }
    pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES; s++) fetch(r_lo + s * AD_ROWS, s, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
    float4 q[GM];
#pragma unroll
    for (int h = 0; h < GM; h++) {
        q[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (h < G && 4 * lane < D) {
            const float4 v = ld4(P.io.q + (int64_t) t * P.io.ldq + (kvh * G + h) * D, 4 * lane);
            q[h] = make_float4(v.x * a.scale, v.y * a.scale, v.z * a.scale, v.w * a.scale);
        }
    }
    // the output entries this CTA finishes
    const int slice = (G * DV + AD_CTAS - 1) / AD_CTAS, mine = rank * slice + tid, oh = mine / DV, od = mine - oh * DV;
    const bool finisher = tid < slice && mine < G * DV;
    float gate = 1.f, sink = 0.f;
    if (finisher) {
        gate = attn_gate(P.io, t, kvh * G + oh, od, DV);
        if (a.sink) sink = attn_sink(P.io, kvh * G + oh);
    }
    const int vh = warp % GM, vp = warp / GM;             // the head and the share of this warp in the value sums
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int r0 = r_lo, it = 0; r0 < r_hi; r0 += AD_ROWS, it++) {
        const int s = it % STAGES, nr = min(AD_ROWS, r_hi - r0);
        const float * K = stage + s * TILE, * V = TIED ? K : K + AD_ROWS * AD_DIM;
        if (it >= STAGES) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
            __syncthreads();
        }
        // scores: rows warp, warp + 8, ...; four rows for all heads are summed over the lanes together
        {
            constexpr int M = 4 * GM, LEFT = 32 / M;
            float v[M];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = warp + AD_WARPS * j;
                const float4 k = i < nr && 4 * lane < D ? *reinterpret_cast<const float4 *>(K + i * AD_DIM + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int h = 0; h < GM; h++) v[h * 4 + j] = fmaf(q[h].w, k.w, fmaf(q[h].z, k.z, fmaf(q[h].y, k.y, q[h].x * k.x)));
            }
            joint_sum<M, 16>(v, lane);
            float x = v[0];
#pragma unroll
            for (int o = LEFT / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            const int at = lane / LEFT, i = warp + AD_WARPS * (at & 3), r = r0 + i;
            if (lane % LEFT == 0) {
                bool seen = i < nr;
                if (seen && (a.window > 0 || pi >= a.cache_rows || a.chunk > 0)) {   // which position does row r hold right now?
                    int p = r;
                    if (r >= keep) {
                        const int ip = pi - keep;         // >= 0 because r < used <= pi + 1
                        p = keep + ip - ((ip - (r - keep)) % ring + ring) % ring;
                        if (p < keep) p = -1;
                    }
                    seen = p >= 0 && p <= pi && (a.window <= 0 || pi - p < a.window || p < a.keep_first);
                }
                if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
                S[at >> 2][i] = seen ? x : -INFINITY;
            }
        }
        __syncthreads();
        if (warp < GM) {
            const float x = S[warp][lane], mo = runm[warp], mn = fmaxf(mo, wmax(x));
            const float p = x == -INFINITY ? 0.f : expf(x - mn), c = mo == -INFINITY ? 0.f : expf(mo - mn);
            S[warp][lane] = p;
            const float sum = wsum(p);
            __syncwarp();
            if (lane == 0) { corr[warp] = c; runm[warp] = mn; runl[warp] = runl[warp] * c + sum; }
        }
        __syncthreads();
        if (vp < PARTS) {
            const float c = corr[vh];
            acc = make_float4(acc.x * c, acc.y * c, acc.z * c, acc.w * c);
            if (4 * lane < DV)
#pragma unroll 4
                for (int i = vp; i < nr; i += PARTS) {
                    const float p = S[vh][i];
                    const float4 x = *reinterpret_cast<const float4 *>(V + i * AD_DIM + 4 * lane);
                    if (p != 0.f) acc = make_float4(fmaf(p, x.x, acc.x), fmaf(p, x.y, acc.y), fmaf(p, x.z, acc.z), fmaf(p, x.w, acc.w));
                }
        }
        __syncthreads();                                  // the stage may be overwritten, and the scores
        const int rn = r0 + STAGES * AD_ROWS;
        if (rn < r_hi) { fetch(rn, s, false); fetch(rn, s, true); }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (vp < PARTS) *reinterpret_cast<float4 *>(&sums[vp][vh][4 * lane]) = acc;
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every CTA of the cluster runs
    for (int i = tid; i < G * DV; i += AD_WARPS * 32) {
        const int h = i / DV, d = i - h * DV, dest = i / slice;
        float v = 0.f;
#pragma unroll
        for (int p = 0; p < PARTS; p++) v += sums[p][h][d];
        send(v, &got[rank][i - dest * slice], dest);
    }
    if (tid < AD_CTAS * GM) {
        const int dest = tid / GM, h = tid - dest * GM;
        send(runm[h], &gotm[rank][h], dest);
        send(runl[h], &gotl[rank][h], dest);
    }
    cluster_barrier();
    if (!finisher) return;
    float M = -INFINITY, L = 0.f, o = 0.f;
#pragma unroll
    for (int c = 0; c < AD_CTAS; c++) M = fmaxf(M, gotm[c][oh]);
#pragma unroll
    for (int c = 0; c < AD_CTAS; c++) {
        const float f = gotm[c][oh] == -INFINITY ? 0.f : expf(gotm[c][oh] - M);
        L = fmaf(gotl[c][oh], f, L);
        if (f != 0.f) o = fmaf(got[c][tid], f, o);
    }
    if (a.sink && M != -INFINITY) L += expf(sink - M);
    put((OT *) P.out, (int64_t) t * (a.heads * DV) + (kvh * G + oh) * DV + od, o * (L > 0.f ? 1.f / L : 0.f) * gate);
}

template <typename OT, int GM, bool TIED>
int launch_group(const DecodeParams & P, int entries, cudaStream_t st) {
    static FuncAttrCache cache;
    const cudaError_t e = ensure_dyn_smem(cache, (const void *) k_attn_decode_group<OT, GM, TIED>, AD_BYTES, true);
    if (e != cudaSuccess) return (int) e;
    return ck_launch([&] { launch_dep(k_attn_decode_group<OT, GM, TIED>, dim3(AD_CTAS, (unsigned) P.a.kv_heads, (unsigned) entries), dim3(AD_WARPS * 32), AD_BYTES, st, P); });
}
template <typename OT>
int launch_typed(const DecodeParams & P, int entries, bool tied, cudaStream_t st) {
    const int g = P.a.heads / P.a.kv_heads;
#define PB_GROUP(GM) return tied ? launch_group<OT, GM, true>(P, entries, st) : launch_group<OT, GM, false>(P, entries, st)
    if (g == 1) PB_GROUP(1);
    if (g == 2) PB_GROUP(2);
    if (g <= 4) PB_GROUP(4);
    PB_GROUP(8);
#undef PB_GROUP
}

}  // namespace

int launch_attn_decode_group(const AttnIO & io, const BatchView & b, const AttnParams & a, const float * kcache, const float * vcache, int64_t slot_stride, void * out,
                             int otype, cudaStream_t st) {
    // A layer's step, 16 heads, us, CTAs of 64 rows per (entry, head) and a merge (mixers.cu) / this:
    // 4 kv heads, one sequence: 8 rows 37.4 / 31.0, 130 40.4 / 30.9, 1990 46.4 / 43.6; eight: 53.8 / 46.9, 59.9 / 46.4, 139.5 / 69.6; 32: 106 / 92, 126 / 95
    // 16 kv heads, one sequence: 40.7 / 34.2, 44.0 / 34.1, 50.9 / 49.1; eight: 57.0 / 56.9, 65.4 / 58.9, 149 / 106; 32: 108 / 126, 132 / 135, at 700 rows 232 / 184
    // beside a delta rule, keys that are their own values, one sequence: 49.5 / 47.4, at 1990 rows 53.9 / 55.6; eight: 83.8 / 77.9, 145 / 87
    // So many sequences of ungrouped heads, whose clusters share nothing, stay with the CTAs per head.
    if (a.heads == a.kv_heads && (int64_t) b.n_entries * a.kv_heads > 256) return (int) cudaErrorNotSupported;
    const bool tied = a.tied_v && kcache == vcache && a.vdim == a.dim;
    auto four = [](int64_t n) { return n % 4 == 0; };
    if (a.heads > 8 * a.kv_heads || a.dim > AD_DIM || a.vdim > AD_DIM || !four(a.dim) || !four(a.vdim) || !four(io.k_row) || !four(io.v_row) || !four(io.ldq) || !four(slot_stride) ||
        !at16(io.q) || !at16(kcache) || !at16(vcache) || (a.tied_v && !tied) || b.n_entries > 65535 || a.kv_heads > 65535)
        return (int) cudaErrorNotSupported;
    const DecodeParams P{io, b.slot, b.off, b.pos0, a, kcache, vcache, slot_stride, out};
    return otype == T_BF16 ? launch_typed<__nv_bfloat16>(P, b.n_entries, tied, st) : launch_typed<float>(P, b.n_entries, tied, st);
}

}  // namespace pb
