// prima.cpp_b200/csrc/heads.cu — the steps around a token's heads with a warp to a head: preparation of queries, keys and values (rotation, unit norm, factors, cache
// store) and of a delta rule's inputs, the join of a dual mixer's branches, and the causal convolution in front of the recurrence with four channels a thread.
// The same steps as gated.cu's kernels (attn_prep_rows, delta_prep_rows, k_dual_post, k_causal_conv), which serve what does not fit here: a lane has four
// neighbouring entries of a head, so heads of up to 128 entries, a multiple of four, at 16 bytes.  The launchers answer cudaErrorNotSupported otherwise.
// Bound: bytes of the rows, which are read and written once, and for few tokens the way to L2 and back.
// us, through shared memory or an element a thread / this (alone, from HBM): preparation of 2048 tokens of 16 heads over 4 of 128 32.0 / 18.1, of 512 tokens beside a delta
// rule 13.2 / 7.5, of one token 8.6 / 5.2; join of 512 tokens of 16 + 16 heads, a CTA a head / a warp 20.0 / 8.9; convolution of 512 tokens over 3072 channels 29.2 / 9.0, of
// one token 4.7 / 3.9.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "launch.h"
#include "layers.h"
#include "mixers.cuh"
#include "rows.cuh"

namespace pb {
namespace {

struct HeadPrep {
    float * q; int64_t ldq; float * k; int64_t ldk; const float * v; int64_t ldv;
    const int32_t * slot, * off, * pos0, * entry_of;
    AttnParams a;
    AttnPrep pr;
    float * kcache, * vcache; int64_t slot_stride;
    // delta rule: unit queries and keys, step sizes, decays per head (rq null: no recurrent branch; ra null: decays come from elsewhere)
    float * rq; int64_t ldrq; float * rk; int64_t ldrk; float * beta; int64_t ldb; float * ra; int64_t lda;
    const float * A_log, * dt_bias;
    int r_qk, r_heads, r_dim;
};

// One CTA per token; its warps take the heads in turns, the last ones the value rows, the recurrence's heads and its numbers
__global__ void __launch_bounds__(1024) k_head_prep(const __grid_constant__ HeadPrep P) {
    __shared__ __align__(16) float cs[128];          // cosines and sines of the token's position, in turns
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const AttnParams & a = P.a;
    const AttnPrep & pr = P.pr;
    pdl_trigger();
    // the batch's description was copied in front of the pass: the angles do not wait for the kernel in front
    const int e = P.entry_of[t], n = P.off[e + 1] - P.off[e], p = P.pos0[e] + (t - P.off[e]), pend = P.pos0[e] + n;
    const float fp = (float) p;
    for (int i = threadIdx.x; i < pr.rot_dims / 2; i += blockDim.x) {
        float s, c;
        sincosf(fp * pr.rot_freq[i], &s, &c);
        cs[2 * i] = c * pr.rot_mag;
        cs[2 * i + 1] = s * pr.rot_mag;
    }
    __syncthreads();
    pdl_wait();
    const int D = a.dim, KD = a.kv_heads * D, VD = attn_v_row(a), rd = pr.rot_dims;
    // where the token's rows go in the cache: of the positions that share a ring row only the last one of this entry is stored
    const int keep = min(a.keep_first, a.cache_rows), ring = a.cache_rows - keep;
    const bool stored = p < keep || (ring > 0 && p >= pend - ring);
    const int64_t crow = p < keep ? p : keep + (p - keep) % max(ring, 1);
    float * kd = P.kcache + (int64_t) P.slot[e] * P.slot_stride + crow * KD;
    float * vd = P.vcache + (int64_t) P.slot[e] * P.slot_stride + crow * VD;
    const float ft = pr.q_temp_every > 0.f ? 1.f + pr.q_temp_coef * logf(floorf((fp + 1.f) / pr.q_temp_every) + 1.f) : 1.f;
    const int heads = a.heads + a.kv_heads, copies = (VD + 127) / 128, total = heads + copies + 2 * P.r_qk + (P.r_qk > 0 ? 1 : 0);
    const bool mine = 4 * lane < D;
    for (int task = warp; task < total; task += nw) {
        if (task < heads) {
            const bool is_q = task < a.heads;
            float * hv = is_q ? P.q + (int64_t) t * P.ldq + task * D : P.k + (int64_t) t * P.ldk + (task - a.heads) * D;
            float4 x = mine ? ld4(hv, 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (rd > 0) {
                if (pr.rot_layout == ROT_INTERLEAVED) {
                    if (4 * lane < rd) {
                        const float4 f = *reinterpret_cast<const float4 *>(cs + 4 * lane);   // (cos, sin) of pairs 2 lane and 2 lane + 1
                        x = make_float4(x.x * f.x - x.y * f.y, x.y * f.x + x.x * f.y, x.z * f.z - x.w * f.w, x.w * f.z + x.z * f.w);
                    }
                } else {   // entry i meets entry i + rd / 2: rd / 8 lanes further on
                    const bool low = 4 * lane < rd / 2, high = !low && 4 * lane < rd;
                    const int other = low ? lane + rd / 8 : high ? lane - rd / 8 : lane;
                    const float4 o = make_float4(__shfl_sync(0xffffffffu, x.x, other), __shfl_sync(0xffffffffu, x.y, other), __shfl_sync(0xffffffffu, x.z, other),
                                                 __shfl_sync(0xffffffffu, x.w, other));
                    if (low || high) {
                        const float * f = cs + 8 * (low ? lane : other);
                        const float sg = low ? -1.f : 1.f;
                        x = make_float4(x.x * f[0] + sg * (o.x * f[1]), x.y * f[2] + sg * (o.y * f[3]), x.z * f[4] + sg * (o.z * f[5]), x.w * f[6] + sg * (o.w * f[7]));
                    }
                }
            }
            float inv = 1.f;
            if (pr.norm == QKN_HEAD_UNIT) inv = 1.f / sqrtf(wsum(squares4(x)) / (float) D + pr.eps);
            if (is_q) inv *= pr.q_scale ? pr.q_scale[task] * ft : ft;
            x = make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv);
            if (mine) {
                put4(hv, 4 * lane, x);
                if (!is_q && stored) put4(kd + (task - a.heads) * D, 4 * lane, x);
            }
        } else if (task < heads + copies) {
            const int i = (task - heads) * 128 + 4 * lane;
            if (stored && i < VD) put4(vd, i, ld4(P.v + (int64_t) t * P.ldv, i));
        } else if (task < heads + copies + 2 * P.r_qk) {
            const int hh = task - heads - copies;
            const bool is_q = hh < P.r_qk, in = 4 * lane < P.r_dim;
            float * hv = is_q ? P.rq + (int64_t) t * P.ldrq + hh * P.r_dim : P.rk + (int64_t) t * P.ldrk + (hh - P.r_qk) * P.r_dim;
            const float4 x = in ? ld4(hv, 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float inv = (1.f / sqrtf(wsum(squares4(x)) + 1e-6f)) * (is_q ? 1.f / sqrtf((float) P.r_dim) : 1.f);
            if (in) put4(hv, 4 * lane, make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv));
        } else {
            for (int h = lane; h < P.r_heads; h += 32) {
                float * b = P.beta + (int64_t) t * P.ldb + h;
                *b = sigmoid_f(*b);
                if (!P.ra) continue;
                float * d = P.ra + (int64_t) t * P.lda + h;
                *d = expf(-expf(P.A_log[h]) * softplus_f(*d + P.dt_bias[h]));
            }
        }
    }
}

// One CTA per token: a warp gates an attention head, or divides a recurrence head by its root mean square and applies its weight and gate
template <typename OT>
__global__ void __launch_bounds__(1024) k_join_heads(const float * o, int heads, int vdim, const float * gate, int64_t ldg, int gate_mode, float left_scale,
                                                    const float * y, int r_heads, int r_vdim, const float * r_gate, int64_t ldrg,
                                                    const float * __restrict__ r_w, int r_gate_act, float eps, float right_scale, OT * __restrict__ out, int64_t ldo) {
    pdl_enter();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, i = 4 * lane;
    for (int task = warp; task < heads + r_heads; task += nw) {
        if (task < heads) {
            if (i >= vdim) continue;
            const float4 x = ld4(o + ((int64_t) t * heads + task) * vdim, i);
            const float * g = gate + (int64_t) t * ldg;
            const float gh = gate_mode == 1 ? sigmoid_f(g[task]) * left_scale : left_scale;
            float4 f = make_float4(gh, gh, gh, gh);
            if (gate_mode == 2) {
                const float4 z = ld4(g + (int64_t) task * vdim, i);
                f = make_float4(gh * sigmoid_f(z.x), gh * sigmoid_f(z.y), gh * sigmoid_f(z.z), gh * sigmoid_f(z.w));
            }
            put4(out, (int64_t) t * ldo + task * vdim + i, make_float4(x.x * f.x, x.y * f.y, x.z * f.z, x.w * f.w));
            continue;
        }
        const int h = task - heads;
        const bool in = i < r_vdim;
        float4 x = in ? ld4(y + ((int64_t) t * r_heads + h) * r_vdim, i) : make_float4(0.f, 0.f, 0.f, 0.f), z = x, w = make_float4(1.f, 1.f, 1.f, 1.f);
        if (in && r_gate_act >= 0) z = ld4(r_gate + (int64_t) t * ldrg + (int64_t) h * r_vdim, i);
        if (in && r_w) w = ld4(r_w + (int64_t) h * r_vdim, i);
        const float inv = 1.f / sqrtf(wsum(squares4(x)) / (float) r_vdim + eps);
        if (!in) continue;
        x = make_float4(x.x * inv * w.x, x.y * inv * w.y, x.z * inv * w.z, x.w * inv * w.w);
        if (r_gate_act == 0) x = make_float4(x.x * sigmoid_f(z.x), x.y * sigmoid_f(z.y), x.z * sigmoid_f(z.z), x.w * sigmoid_f(z.w));
        else if (r_gate_act > 0) x = make_float4(x.x * silu_f(z.x), x.y * silu_f(z.y), x.z * silu_f(z.z), x.w * silu_f(z.w));
        put4(out, (int64_t) t * ldo + (int64_t) heads * vdim + (int64_t) h * r_vdim + i, make_float4(x.x * right_scale, x.y * right_scale, x.z * right_scale, x.w * right_scale));
    }
}

// convolution of four taps: a thread takes four channels of TOK tokens
template <int TOK>
__global__ void __launch_bounds__(128) k_conv4(const float * u, int64_t ldu, const int32_t * __restrict__ slot, const int32_t * __restrict__ off,
                                               const int32_t * __restrict__ entry_of, int n_tokens, int channels, const float * __restrict__ w, int silu_from,
                                               float * conv_state, int64_t slot_stride, float * out, int64_t ldo, int advance) {
    const int c = 4 * (blockIdx.x * 128 + threadIdx.x);
    float4 wc[4];                                    // a channel's taps, the oldest input's first
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < 4; i++) wc[i] = c < channels ? ld4(w, 4 * (int64_t) (c + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
    pdl_wait();
    if (c >= channels) return;
#pragma unroll
    for (int j = 0; j < TOK; j++) {
        const int t = blockIdx.y * TOK + j;
        if (t >= n_tokens) break;
        const int e = entry_of[t], lt = t - off[e];
        float * st = conv_state + (int64_t) slot[e] * slot_stride + c;   // [3][channels], row 2 = the input just before this entry
        float4 in[4];
#pragma unroll
        for (int d = 0; d < 4; d++) in[d] = lt - 3 + d >= 0 ? ld4(u, (int64_t) (t - 3 + d) * ldu + c) : ld4(st, (int64_t) (lt + d) * channels);
        float r[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float x[4] = {(&in[0].x)[i], (&in[1].x)[i], (&in[2].x)[i], (&in[3].x)[i]};
            r[i] = fmaf(wc[i].w, x[3], fmaf(wc[i].z, x[2], fmaf(wc[i].y, x[1], wc[i].x * x[0])));
            if (c + i >= silu_from) r[i] = silu_f(r[i]);
        }
        put4(out, (int64_t) t * ldo + c, make_float4(r[0], r[1], r[2], r[3]));
        if (advance) {   // entries of one token: this thread is the only reader and writer of its channels' state
#pragma unroll
            for (int d = 0; d < 3; d++) put4(st, (int64_t) d * channels, in[d + 1]);
        }
    }
}

bool head_ok(int dim) { return dim > 0 && dim % 4 == 0 && dim <= 128; }
bool rows_ok(const void * p, int64_t ld) { return at16(p) && ld % 4 == 0; }
// a token's tasks over as many warps as it takes when tokens are few
int head_threads(int n_tokens, int tasks) { return n_tokens >= 128 ? 256 : 32 * (tasks < 32 ? tasks : 32); }

}  // namespace

int launch_head_prep(float * rq, int64_t ldrq, float * rk, int64_t ldrk, float * beta, int64_t ldb, float * ra, int64_t lda, const float * A_log, const float * dt_bias, int r_qk,
                     int r_heads, int r_dim, float * q, int64_t ldq, float * k, int64_t ldk, const float * v, int64_t ldv, const BatchView & b, const AttnParams & a, const AttnPrep & pr,
                     float * kcache, float * vcache, int64_t slot_stride, cudaStream_t st) {
    const bool rot_ok = pr.rot_dims == 0 || (pr.rot_layout == ROT_INTERLEAVED ? pr.rot_dims % 4 == 0 : pr.rot_dims % 8 == 0);
    const int vd = attn_v_row(a);
    if (!head_ok(a.dim) || !rot_ok || pr.v_rot || pr.norm == QKN_WHOLE_WEIGHT || !rows_ok(q, ldq) || (a.kv_heads > 0 && (!rows_ok(k, ldk) || !rows_ok(kcache, slot_stride))) ||
        (vd > 0 && (vd % 4 != 0 || !rows_ok(v, ldv) || !rows_ok(vcache, slot_stride))) || (rq && (!head_ok(r_dim) || !rows_ok(rq, ldrq) || !rows_ok(rk, ldrk))))
        return (int) cudaErrorNotSupported;
    const HeadPrep P{q, ldq, k, ldk, v, ldv, b.slot, b.off, b.pos0, b.entry_of, a, pr, kcache, vcache, slot_stride, rq, ldrq, rk, ldrk, beta, ldb, ra, lda, A_log, dt_bias,
                     rq ? r_qk : 0, r_heads, r_dim};
    const int tasks = a.heads + a.kv_heads + (vd + 127) / 128 + (rq ? 2 * r_qk + 1 : 0);
    return ck_launch([&] { launch_dep(k_head_prep, dim3((unsigned) b.n_tokens), dim3((unsigned) head_threads(b.n_tokens, tasks)), 0, st, P); });
}
int launch_join_heads(const float * o, int n_tokens, int heads, int vdim, const float * gate, int64_t ldg, int gate_mode, float left_scale, const float * y, int r_heads, int r_vdim,
                      const float * r_gate, int64_t ldrg, const float * r_w, int r_gate_act, float eps, float right_scale, void * out, int64_t ldo, int otype, cudaStream_t st) {
    if (!head_ok(vdim) || !head_ok(r_vdim) || !at16(o) || !at16(y) || !at16(r_w) || !rows_ok(out, ldo) || (gate_mode == 2 && !rows_ok(gate, ldg)) ||
        (r_gate_act >= 0 && !rows_ok(r_gate, ldrg)))
        return (int) cudaErrorNotSupported;
    const dim3 block((unsigned) head_threads(n_tokens, heads + r_heads));
    return ck_launch([&] {
        if (otype == T_BF16)
            launch_dep(k_join_heads<__nv_bfloat16>, dim3((unsigned) n_tokens), block, 0, st, o, heads, vdim, gate, ldg, gate_mode, left_scale, y, r_heads, r_vdim, r_gate, ldrg, r_w,
                       r_gate_act, eps, right_scale, (__nv_bfloat16 *) out, ldo);
        else
            launch_dep(k_join_heads<float>, dim3((unsigned) n_tokens), block, 0, st, o, heads, vdim, gate, ldg, gate_mode, left_scale, y, r_heads, r_vdim, r_gate, ldrg, r_w, r_gate_act, eps,
                       right_scale, (float *) out, ldo);
    });
}
int launch_conv4(const float * u, int64_t ldu, const BatchView & b, int channels, const float * w, int silu_from, float * conv_state, int64_t slot_stride, float * out, int64_t ldo,
                 int advance, cudaStream_t st) {
    if (channels % 4 != 0 || !rows_ok(u, ldu) || !at16(w) || !rows_ok(conv_state, slot_stride) || !rows_ok(out, ldo)) return (int) cudaErrorNotSupported;
    const unsigned tiles = (unsigned) ((channels / 4 + 127) / 128);
    if ((b.n_tokens + 3) / 4 > 65535) return (int) cudaErrorNotSupported;   // a grid's second dimension: more tokens go to the general kernel
    return ck_launch([&] {
        // Four tokens a thread share the weights and, in L1, the inputs, but a quarter of the CTAs keep the SMs busy only from so many on.  us of the convolution and its
        // state's step, a token a thread / four: 3072 channels 128 tokens 13.1 / 14.9, 256 tokens 15.2 / 15.2, 384 tokens 15.3 / 15.2, 512 tokens 17.2 / 15.7; 2048 channels
        // 256 tokens 13.4 / 13.9, 512 tokens 15.6 / 15.4, 1024 tokens 19.6 / 17.1
        if ((int64_t) b.n_tokens * tiles >= 14 * sm_count())
            launch_dep(k_conv4<4>, dim3(tiles, (unsigned) ((b.n_tokens + 3) / 4)), dim3(128), 0, st, u, ldu, b.slot, b.off, b.entry_of, b.n_tokens, channels, w, silu_from, conv_state,
                       slot_stride, out, ldo, advance);
        else
            launch_dep(k_conv4<1>, dim3(tiles, (unsigned) b.n_tokens), dim3(128), 0, st, u, ldu, b.slot, b.off, b.entry_of, b.n_tokens, channels, w, silu_from, conv_state, slot_stride, out,
                       ldo, advance);
    });
}

}  // namespace pb
