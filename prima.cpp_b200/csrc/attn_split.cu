// prima.cpp_b200/csrc/attn_split.cu — prompt attention of the layer-list models (windows, kept first tokens, chunks, soft-cap, sinks, gates, grouped
// heads, keys with a shared tail, another layer's cache) on the 5th-generation tensor cores, with fp32 inputs kept to 22 bits and more:
// every fp32 operand x is two f16 numbers, hi = f16(x s) and lo = f16(x s - hi) with s a power of two per row that puts the row's largest
// entry between 2^13 and 2^14, and a product is lo hi + hi lo + hi hi with fp32 accumulation, the small products first.  What is dropped (lo lo and
// the rounding of lo) is 2^-22 of the row's entries and less.  A softmax weight takes its value row's power of two along: the largest such product
// that a query has in a key tile comes to 2^14, or, in a tile that every query of the CTA sees and whose values lie within 2^12 of one another,
// the tile's largest value does.  So what a query does not see, however large, or no number at all, does not touch its row.  Scores, softmax, its
// running maximum and sum and the weighted sum across key tiles stay in fp32 registers.
// Two launches: k_split_kv writes keys and values once, split and laid out as the operands' shared-memory images; k_attn_split walks them.
// Only models that compute in bf16 come here (the result is rounded to 2^-9 next); float32 models keep the fp32 FMA kernels of mixers.cu.
// Against float64 in models where nothing else rounds below fp32, six kinds of attention (windows, chunks, sinks, caps, gates, shared key tails), head
// sizes 64 and 128, 40 to 300 keys, three seeds: 2.8e-7 .. 5.6e-7 off, 0.96 to 1.02 times the FMA kernel, 0.99 over all.
// Measured with the split pass, FMA kernel -> these: 2048 tokens, 16 heads of 128 over 4, causal 1516 -> 94 us; 512 tokens 176 -> 37; latent heads,
// prompts of 1111, 300 and 77 tokens 522 -> 84.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "launch.h"
#include "layers.h"
#include "mixers.cuh"
#include "tc.cuh"

namespace pb {
namespace {

constexpr int SP_KEYS = 128;                   // positions of a key tile
constexpr int SP_K_UNIT = 2 * SP_KEYS * 128;   // 64 head entries of a tile's keys: hi, lo, each 128 rows of 128 bytes
constexpr int SP_MAX_ND = 3, SP_MAX_NV = 2;    // head sizes up to 192, value sizes up to 128
// of a tile: key scales [128], value scales relative to the tile's largest [128], value exponents [128], [4]: some value is no number; exponents
// are far apart; the largest value scale
constexpr int SP_SCALES = 1552, SP_SPREAD = 12;
constexpr int SP_SLOT = 16384, SP_MAX_SLOTS = 11;   // the ring's pieces: hi or lo of a unit
constexpr int SP_THREADS = 384, SP_SM_THREADS = 256;
// registers: 168 a thread at the launch, 128 x 88 + 256 x 208 of the same 64512 from the roles on
constexpr int SP_REGS_FEW = 88, SP_REGS_SM = 208;
static_assert(128 * SP_REGS_FEW + SP_SM_THREADS * SP_REGS_SM <= SP_THREADS * 168);

__host__ __device__ inline int sp_v_unit(int nv) { return 2 * nv * 64 * 128; }   // 64 positions of a tile's values: hi, lo, each nv blocks of 64 rows of 128 bytes
__host__ __device__ inline int64_t sp_tile_bytes(int nd, int nv) { return (int64_t) nd * SP_K_UNIT + 2 * sp_v_unit(nv) + SP_SCALES; }

struct SplitParams {
    AttnIO io;
    AttnParams a;
    const int32_t * off;
    uint8_t * ws;              // [kv head][tile slot][sp_tile_bytes]; entry e's first slot: off[e] / 128 + e
    int slots, kv_first;       // kv heads go through the scratch in groups: this launch's first one
    void * out;
    int nd, nv, gqa, tok_per_cta, slots_ring;
    int * abort_flag;
};

constexpr uint32_t NO_NUMBER = 0x7f800000u;   // bits of a magnitude from here on: an infinity or a NaN
__device__ __forceinline__ uint32_t magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }
// largest magnitude of the numbers in a warp's row, for rows whose plain maximum is none
template <int N>
__device__ __forceinline__ uint32_t max_number(const float (&x)[N][2]) {
    uint32_t m = 0u;
#pragma unroll
    for (int c = 0; c < N; c++)
#pragma unroll
        for (int i = 0; i < 2; i++)
            if (magnitude(x[c][i]) < NO_NUMBER) m = max(m, magnitude(x[c][i]));
    return __reduce_max_sync(0xffffffffu, m);
}
// power of two that puts the largest entry (bits of its magnitude) in [2^13, 2^14); e: the clamped exponent it follows from
__device__ __forceinline__ float split_scale(uint32_t max_bits, int lowest, int & e) {
    e = min(max((int) (max_bits >> 23), lowest), 254);
    return __uint_as_float((uint32_t) max(267 - e, 1) << 23);
}
__device__ __forceinline__ void split2(float x, float y, uint32_t & hi, uint32_t & lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

// One CTA: a tile of 128 positions of one kv head and entry; a warp takes a position at a time, a lane two neighbouring entries of every 64.
__global__ void __launch_bounds__(256, 2) k_split_kv(const __grid_constant__ SplitParams P) {
    __shared__ int ev[SP_KEYS];        // exponents, -: the row holds something that is no number, 0: nothing but zeros
    pdl_enter();
    const int e = blockIdx.z, kvh = P.kv_first + blockIdx.y, tile = blockIdx.x;
    const int t_begin = P.off[e], n = P.off[e + 1] - t_begin;
    if (tile * SP_KEYS >= n) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const AttnIO & io = P.io;
    const int D = P.a.dim, DN = P.a.dim - P.a.shared_dim, DV = P.a.vdim;
    const int64_t at = io.kv_slot ? (int64_t) io.kv_slot[e] * io.kv_slot_stride : 0;
    const float * kb = io.k + (io.kv_slot ? at : (int64_t) t_begin * io.ldk) + (int64_t) kvh * DN;
    const float * vb = io.v + (io.kv_slot ? at : (int64_t) t_begin * io.ldv) + (int64_t) kvh * DV;
    const float * ks = io.ks ? io.ks + (int64_t) t_begin * io.ldks : nullptr;
    uint8_t * dst = P.ws + ((int64_t) blockIdx.y * P.slots + t_begin / SP_KEYS + e + tile) * sp_tile_bytes(P.nd, P.nv);
    uint8_t * dv = dst + P.nd * SP_K_UNIT;
    float * sc = reinterpret_cast<float *>(dv + 2 * sp_v_unit(P.nv));
    const int blk_b = sp_v_unit(P.nv) / 2;                         // the lo half of a unit of values
    constexpr int ROWS = 4;
    int bad = 0;
    for (int r0 = warp * 16; r0 < warp * 16 + 16; r0 += ROWS) {
        float k[ROWS][SP_MAX_ND][2], v[ROWS][SP_MAX_NV][2];
#pragma unroll
        for (int j = 0; j < ROWS; j++) {
            const int64_t p = (int64_t) tile * SP_KEYS + r0 + j;
            const bool live = p < n;
#pragma unroll
            for (int c = 0; c < SP_MAX_ND; c++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int d = 64 * c + 2 * lane + i;
                    k[j][c][i] = live && d < D ? (d < DN ? kb[p * io.ldk + d] : ks[p * io.ldks + d - DN]) : 0.f;
                }
#pragma unroll
            for (int c = 0; c < SP_MAX_NV; c++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int d = 64 * c + 2 * lane + i;
                    v[j][c][i] = live && d < DV ? vb[p * io.ldv + d] : 0.f;
                }
        }
        uint32_t mk[ROWS], mv[ROWS], worst = 0u;
#pragma unroll
        for (int j = 0; j < ROWS; j++) {
            mk[j] = mv[j] = 0u;
#pragma unroll
            for (int c = 0; c < SP_MAX_ND; c++)
#pragma unroll
                for (int i = 0; i < 2; i++) mk[j] = max(mk[j], magnitude(k[j][c][i]));
#pragma unroll
            for (int c = 0; c < SP_MAX_NV; c++)
#pragma unroll
                for (int i = 0; i < 2; i++) mv[j] = max(mv[j], magnitude(v[j][c][i]));
            mk[j] = __reduce_max_sync(0xffffffffu, mk[j]);
            mv[j] = __reduce_max_sync(0xffffffffu, mv[j]);
            worst = max(worst, max(mk[j], mv[j]));
        }
        uint32_t odd = 0u;   // bit j: a key of row j is no number, bit ROWS + j: a value
        if (worst >= NO_NUMBER) {
#pragma unroll
            for (int j = 0; j < ROWS; j++) {
                if (mk[j] >= NO_NUMBER) { mk[j] = max_number(k[j]); odd |= 1u << j; }
                if (mv[j] >= NO_NUMBER) {   // such values stay out of the products (a weight of zero does not silence them): k_attn_split puts them in
                    mv[j] = max_number(v[j]);
                    odd |= 1u << (ROWS + j);
                    bad = 1;
#pragma unroll
                    for (int c = 0; c < SP_MAX_NV; c++)
#pragma unroll
                        for (int i = 0; i < 2; i++)
                            if (magnitude(v[j][c][i]) >= NO_NUMBER) v[j][c][i] = 0.f;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < ROWS; j++) {
            const int r = r0 + j;
            int ek, e_v;
            const float sk = split_scale(mk[j], 14, ek), sv = split_scale(mv[j], 28, e_v);
            const uint32_t in_row = (uint32_t) ((((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4);
#pragma unroll
            for (int c = 0; c < SP_MAX_ND; c++)
                if (c < P.nd) {
                    uint32_t hi, lo;
                    split2(k[j][c][0] * sk, k[j][c][1] * sk, hi, lo);
                    uint8_t * o = dst + c * SP_K_UNIT + (r >> 3) * 1024 + (r & 7) * 128 + in_row;
                    *reinterpret_cast<uint32_t *>(o) = hi;
                    *reinterpret_cast<uint32_t *>(o + SP_K_UNIT / 2) = lo;
                }
            const int rv = r & 63;
#pragma unroll
            for (int c = 0; c < SP_MAX_NV; c++)
                if (c < P.nv) {
                    uint32_t hi, lo;
                    split2(v[j][c][0] * sv, v[j][c][1] * sv, hi, lo);
                    uint8_t * o = dv + (r >> 6) * sp_v_unit(P.nv) + c * 8192 + (rv >> 3) * 1024 + (rv & 7) * 128 + in_row;
                    *reinterpret_cast<uint32_t *>(o) = hi;
                    *reinterpret_cast<uint32_t *>(o + blk_b) = lo;
                }
            if (lane == 0) {
                sc[r] = __uint_as_float((uint32_t) (ek - 13) << 23);
                sc[2 * SP_KEYS + r] = (float) (e_v - 127);
                ev[r] = (odd >> (ROWS + j)) & 1u ? -e_v : mv[j] ? e_v : 0;
            }
            if ((odd >> j) & 1u) {   // an infinity or a NaN goes into lo alone: a score is then what its sign makes of it
#pragma unroll
                for (int c = 0; c < SP_MAX_ND; c++)
                    if (c < P.nd) {
                        const float x = k[j][c][0] * sk, y = k[j][c][1] * sk, fx = fabsf(x) < INFINITY ? x : 0.f, fy = fabsf(y) < INFINITY ? y : 0.f;
                        uint32_t hi, lo;
                        split2(fx, fy, hi, lo);
                        const __half2 l = __floats2half2_rn(x, y);
                        const uint32_t raw = *reinterpret_cast<const uint32_t *>(&l);
                        if (fx != x) lo = (lo & 0xffff0000u) | (raw & 0xffffu);
                        if (fy != y) lo = (lo & 0xffffu) | (raw & 0xffff0000u);
                        uint8_t * o = dst + c * SP_K_UNIT + (r >> 3) * 1024 + (r & 7) * 128 + in_row;
                        *reinterpret_cast<uint32_t *>(o) = hi;
                        *reinterpret_cast<uint32_t *>(o + SP_K_UNIT / 2) = lo;
                    }
            }
        }
    }
    bad = __syncthreads_or(bad);
    // the values' powers of two meet the weights: relative to the tile's largest one, times 2^14 (weights are at most 1, f16 reaches 2^16)
    if (warp < 4) {
        int top = 28, low = 254;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int e_v = abs(ev[32 * i + lane]);
            top = max(top, e_v);
            low = min(low, e_v ? e_v : 254);
        }
        top = __reduce_max_sync(0xffffffffu, top);
        low = __reduce_min_sync(0xffffffffu, low);
        const int r = warp * 32 + lane, f = 141 + max(abs(ev[r]), 28) - top;
        sc[SP_KEYS + r] = __uint_as_float((f >= 1 ? (uint32_t) f << 23 : 0u) | (ev[r] < 0 ? 0x80000000u : 0u));   // sign: something that is no number
        if (r < 4) sc[3 * SP_KEYS + r] = r == 0 ? (bad ? 1.f : 0.f) : r == 1 ? (top - low > SP_SPREAD ? 1.f : 0.f) : __uint_as_float((uint32_t) (top - 27) << 23);
    }
}

struct SpCtl {
    uint64_t full[SP_MAX_SLOTS], empty[SP_MAX_SLOTS], sc_full[2], sc_empty[2], s_full[2], p_full[2], o_full[2], o_free[2];
    uint32_t tmem_base;
    int abort;
    float2 row_max[2][2][128];     // [tile parity][half of the keys][row]: largest score, largest exponent of weight x value scale
    float q_scale[128];
    float row_l[2][128];
    alignas(16) float ones[64];
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void * src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// what column d of the values a query sees holds besides numbers, added up (0: nothing).  tiles: the entry's and kv head's first split tile
__device__ __noinline__ float not_numbers(const SplitParams & P, const uint8_t * tiles, int e, int kvh, int qi, int d) {
    const AttnIO & io = P.io;
    const int64_t tile_bytes = sp_tile_bytes(P.nd, P.nv), row0 = io.kv_slot ? 0 : P.off[e];
    const float * vb = io.v + (io.kv_slot ? (int64_t) io.kv_slot[e] * io.kv_slot_stride : row0 * io.ldv) + (int64_t) kvh * P.a.vdim + d;
    const int lo = attn_first_visible(P.a, qi);
    float sum = 0.f;
    for (int tile = 0; tile * SP_KEYS <= qi; tile++) {
        const float * sc = reinterpret_cast<const float *>(tiles + tile * tile_bytes + P.nd * SP_K_UNIT + 2 * sp_v_unit(P.nv));
        if (sc[3 * SP_KEYS] == 0.f) continue;
        for (int r = 0; r < SP_KEYS; r++) {
            const int j = tile * SP_KEYS + r;
            if (j <= qi && (j >= lo || j < P.a.keep_first) && (__float_as_uint(sc[SP_KEYS + r]) >> 31)) {
                const float v = vb[(int64_t) j * io.ldv];
                if (!(fabsf(v) < INFINITY)) sum += v;
            }
        }
    }
    return sum;
}
// 2^d for an integer d <= 0 (0 from 2^-127 on, and for what is no number)
__device__ __forceinline__ float pow2_down(float d) { return d > -126.5f ? __uint_as_float((uint32_t) (127 + (int) d) << 23) : 0.f; }
// the n low ones of 64 bits
__device__ __forceinline__ uint64_t below(int n) { return n >= 64 ? ~0ull : n <= 0 ? 0ull : (1ull << n) - 1; }
__device__ __forceinline__ float gate_factor(const AttnIO & io, int64_t row, int h, int d, int DV) {
    if (io.gate_mode == 1) return sigmoid_f(io.gate[row * io.ldg + h]);
    if (io.gate_mode == 2) return sigmoid_f(io.gate[row * io.ldg + (int64_t) h * DV + d]);
    return 1.f;
}

// One CTA: 128 query rows (the heads of a GQA group x 128 / group consecutive tokens) of one entry and kv head.  Tensor memory: S twice (2 x 128
// columns; the split weights go over the scores they come from), the tile's weighted sum twice (2 x 128).
//   warp 0       lo and hi pieces of key units (64 head entries of 128 keys, 16 KB each) and value units (64 positions) by bulk copies of the split
//                images; the first ones arrive while the others split the queries
//   warp 1       MMA issuer, owner of the tensor memory; S(j + 1) goes before P(j) V(j)
//   warps 4 - 11 softmax: thread = (row, half of the tile's keys); the weighted sum [row][half of the value columns] in registers.  64 scores and
//                64 sums a thread do not fit the 168 registers of twelve warps (180 bytes went through local memory once a tile): the other warpgroup
//                gives up 80 of its own
// Bound: in the steady state S takes 1900 and P V 2500 clocks of the tensor cores (24 MMAs each), the softmax warps 4200 beside them, and a tile
// 4400 to 4600.  It took 7300 to 8200 while every score was tested against the mask (2500 of them) and a unit's memory came free only behind all
// of its products (900 of waiting for copies).  A CTA that is the first on its SM loses about 13000 clocks more to code that is not there yet.
// Measured in one run, start to end: 2048 tokens, 16 heads of 128 over 4, causal 119 -> 91 us; 512 tokens 45 -> 31; the latent prompts above 95 -> 77.
template <typename OT, bool CAP>
__global__ void __launch_bounds__(SP_THREADS, 1) k_attn_split(const __grid_constant__ SplitParams P) {
    extern __shared__ uint8_t smem_raw[];
    const AttnIO & io = P.io;
    const AttnParams & a = P.a;
    const int e = blockIdx.z, kvh = P.kv_first + blockIdx.x;
    const int t_begin = P.off[e], n = P.off[e + 1] - t_begin;                     // of the batch's description, copied in front of the pass
    const int q0 = ((int) gridDim.y - 1 - (int) blockIdx.y) * P.tok_per_cta;      // long rows first
    if (q0 >= n) return;
    const int toks = min(P.tok_per_cta, n - q0), rows = toks * P.gqa;
    uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int nd = P.nd, nv = P.nv, slots = P.slots_ring, v_unit = sp_v_unit(nv), q_piece = nd * 16384;
    uint8_t * q_s = smem, * ring = smem + 2 * q_piece;                            // queries: hi, lo, each nd blocks of 128 rows of 128 bytes
    float * scales = reinterpret_cast<float *>(ring + slots * SP_SLOT);       // [2][SP_SCALES]
    SpCtl * ctl = reinterpret_cast<SpCtl *>(ring + slots * SP_SLOT + 2 * SP_SCALES);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    volatile int * cta_abort = &ctl->abort;
    // key tiles some row sees: the kept first tokens' ones, then from the window's (chunk's) first position to the last query
    const int w_lo = attn_first_visible(a, q0), s_hi = min(a.keep_first, w_lo);
    const int kept = (s_hi + SP_KEYS - 1) / SP_KEYS, first = max(w_lo / SP_KEYS, kept), last = (q0 + toks - 1) / SP_KEYS;
    const int nt = kept + last - first + 1;
    auto tile_of = [&](int j) { return j < kept ? j : first + j - kept; };

    if (threadIdx.x == 0) {
        for (int i = 0; i < SP_MAX_SLOTS; i++) { mbar_init(&ctl->full[i], 1); mbar_init(&ctl->empty[i], 1); }
        for (int i = 0; i < 2; i++) {
            mbar_init(&ctl->sc_full[i], 1); mbar_init(&ctl->sc_empty[i], 8); mbar_init(&ctl->s_full[i], 1); mbar_init(&ctl->p_full[i], 8);
            mbar_init(&ctl->o_full[i], 1); mbar_init(&ctl->o_free[i], 8);
        }
        ctl->abort = 0;
        mbar_fence_init();
    }
    if (threadIdx.x < 64) ctl->ones[threadIdx.x] = 1.f;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        pdl_trigger();   // behind the allocation: a later kernel's CTA on this SM must not take the columns first and wait for this one
    }
    __syncthreads();
    pdl_wait();          // queries and the split images are the kernels' in front
    if (warp >= 4) {
        const int w = warp - 4, D = a.dim;
        for (int r0 = w * 16; r0 < w * 16 + 16; r0 += 4) {
            float x[4][SP_MAX_ND][2];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int r = r0 + j;
                const float * src = io.q + (int64_t) (t_begin + q0 + r / P.gqa) * io.ldq + (int64_t) (kvh * P.gqa + r % P.gqa) * D;
#pragma unroll
                for (int c = 0; c < SP_MAX_ND; c++)
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const int d = 64 * c + 2 * lane + i;
                        x[j][c][i] = r < rows && d < D ? src[d] : 0.f;
                    }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int r = r0 + j;
                uint32_t m = 0u;
#pragma unroll
                for (int c = 0; c < SP_MAX_ND; c++)
#pragma unroll
                    for (int i = 0; i < 2; i++) m = max(m, magnitude(x[j][c][i]));
                m = __reduce_max_sync(0xffffffffu, m);
                int eq;
                const float s = split_scale(m, 14, eq);
#pragma unroll
                for (int c = 0; c < SP_MAX_ND; c++)
                    if (c < nd) {
                        uint32_t hi, lo;
                        split2(x[j][c][0] * s, x[j][c][1] * s, hi, lo);
                        uint8_t * o = q_s + c * 16384 + (r >> 3) * 1024 + (r & 7) * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4;
                        *reinterpret_cast<uint32_t *>(o) = hi;
                        *reinterpret_cast<uint32_t *>(o + q_piece) = lo;
                    }
                if (lane == 0) ctl->q_scale[r] = __uint_as_float((uint32_t) (eq - 13) << 23);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1 || warp >= 4) {      // the first keys are on their way while the queries are split
        fence_before();
        asm volatile("bar.sync 2, %0;" ::"n"(SP_SM_THREADS + 32) : "memory");
        fence_after();
    }
    const uint32_t tmem = *(volatile uint32_t *) &ctl->tmem_base;
    constexpr uint32_t O0 = 256;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SP_REGS_FEW));
        if (warp == 0) {
            const uint8_t * src0 = P.ws + ((int64_t) blockIdx.x * P.slots + t_begin / SP_KEYS + e) * sp_tile_bytes(nd, nv);
            int slot = 0;
            uint32_t turn = 0u;                             // parity of the round in which the ring is filled
            bool wrapped = false;
            auto load = [&](const uint8_t * src, uint32_t bytes) {
                if (wrapped) mbar_wait(&ctl->empty[slot], turn ^ 1u, cta_abort, P.abort_flag);
                __syncwarp();
                if (elect_one()) {
                    mbar_arrive_expect_tx(&ctl->full[slot], bytes);
                    bulk_load(smem_u32(ring + slot * SP_SLOT), src, bytes, smem_u32(&ctl->full[slot]));
                }
                __syncwarp();
                if (++slot == slots) { slot = 0; turn ^= 1u; wrapped = true; }
            };
            for (int j = 0; j <= nt && !*cta_abort; j++) {   // K(0) K(1) V(0) K(2) V(1) ...
                if (j < nt) {
                    const uint8_t * src = src0 + (int64_t) tile_of(j) * sp_tile_bytes(nd, nv);
                    if (j >= 2) mbar_wait(&ctl->sc_empty[j & 1], (uint32_t) ((j / 2 - 1) & 1), cta_abort, P.abort_flag);
                    __syncwarp();
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&ctl->sc_full[j & 1], SP_SCALES);
                        bulk_load(smem_u32(scales) + (j & 1) * SP_SCALES, src + nd * SP_K_UNIT + 2 * v_unit, SP_SCALES, smem_u32(&ctl->sc_full[j & 1]));
                    }
                    __syncwarp();
                    for (int p = 1; p >= 0; p--)            // lo of all units, then hi
                        for (int c = 0; c < nd; c++) load(src + c * SP_K_UNIT + p * (SP_K_UNIT / 2), SP_K_UNIT / 2);
                }
                if (j > 0) {
                    const uint8_t * src = src0 + (int64_t) tile_of(j - 1) * sp_tile_bytes(nd, nv) + nd * SP_K_UNIT;
                    for (int p = 1; p >= 0; p--)
                        for (int c = 0; c < 2; c++) load(src + c * v_unit + p * (v_unit / 2), (uint32_t) v_unit / 2);
                }
            }
            __syncwarp();
        } else if (warp == 1) {
            constexpr uint32_t idesc = (1u << 4) | ((uint32_t) (SP_KEYS >> 3) << 17) | ((uint32_t) (128 >> 4) << 24);
            const uint32_t idesc_v = (1u << 4) | (1u << 16) | ((uint32_t) (nv * 64 >> 3) << 17) | ((uint32_t) (128 >> 4) << 24);
            const uint64_t dq = desc_sw128(smem_u32(q_s));
            const uint32_t q_lo = (uint32_t) (q_piece >> 4);
            const bool leader = elect_one();
            int slot = 0;
            uint32_t turn = 0u;
            // the next piece of the ring, arrived
            auto next = [&]() {
                const int at = slot;
                mbar_wait(&ctl->full[at], turn, cta_abort, P.abort_flag);
                __syncwarp();
                if (++slot == slots) { slot = 0; turn ^= 1u; }
                return at;
            };
            // the small products of all units go first: what the tensor cores cut off at each step is a share of the sum so far; lo pieces before hi, so
            // that their memory takes the next piece two thirds of the products earlier
            auto scores = [&](int j) {
                const uint32_t d = tmem + (uint32_t) ((j & 1) * 128);
                int at[SP_MAX_ND];
                for (int c = 0; c < nd; c++) {
                    const int s = next();
                    const uint64_t lk = desc_sw128(smem_u32(ring + s * SP_SLOT)), hq = dq + c * (16384 >> 4);
                    if (c == 0) fence_after();
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < 4; k++) mma_f16<1>(d, hq + 2 * k, lk + 2 * k, idesc, (uint32_t) ((c | k) != 0));
                        mma_commit(&ctl->empty[s]);
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int c = 0; c < SP_MAX_ND; c++) {
                    if (c >= nd) break;
                    at[c] = next();
                    const uint64_t hk = desc_sw128(smem_u32(ring + at[c] * SP_SLOT)), lq = dq + c * (16384 >> 4) + q_lo;
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < 4; k++) mma_f16<1>(d, lq + 2 * k, hk + 2 * k, idesc, 1u);
                    }
                    __syncwarp();
                }
                if (leader) {
#pragma unroll
                    for (int c = 0; c < SP_MAX_ND; c++) {
                        if (c >= nd) break;
                        const uint64_t hk = desc_sw128(smem_u32(ring + at[c] * SP_SLOT)), hq = dq + c * (16384 >> 4);
#pragma unroll
                        for (int k = 0; k < 4; k++) mma_f16<1>(d, hq + 2 * k, hk + 2 * k, idesc, 1u);
                        mma_commit(&ctl->empty[at[c]]);
                    }
                    mma_commit(&ctl->s_full[j & 1]);
                }
                __syncwarp();
            };
            scores(0);
            for (int j = 0; j < nt && !*cta_abort; j++) {
                if (j + 1 < nt) scores(j + 1);       // its columns held P(j - 1), whose products precede it in the pipe
                const int buf = j & 1;
                mbar_wait(&ctl->p_full[buf], (uint32_t) ((j / 2) & 1), cta_abort, P.abort_flag);
                if (j >= 2) mbar_wait(&ctl->o_free[buf], (uint32_t) ((j / 2 - 1) & 1), cta_abort, P.abort_flag);
                __syncwarp();
                fence_after();
                const uint32_t d = tmem + O0 + (uint32_t) (buf * 128), p0 = tmem + (uint32_t) (buf * 128);      // 16 columns hi, 16 columns lo of 32 keys, then the next 32
                int at[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int s = next();
                    const uint64_t lv = desc_sw128_mn(smem_u32(ring + s * SP_SLOT), 8192);
                    const uint32_t p = p0 + (uint32_t) (h * 64);
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < 4; k++) mma_f16_ts(d, p + (k >> 1) * 32 + (k & 1) * 8, lv + k * (2048 >> 4), idesc_v, (uint32_t) ((h | k) != 0));
                        mma_commit(&ctl->empty[s]);
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    at[h] = next();
                    const uint64_t hv = desc_sw128_mn(smem_u32(ring + at[h] * SP_SLOT), 8192);
                    const uint32_t p = p0 + (uint32_t) (h * 64);
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < 4; k++) mma_f16_ts(d, p + (k >> 1) * 32 + 16 + (k & 1) * 8, hv + k * (2048 >> 4), idesc_v, 1u);
                    }
                    __syncwarp();
                }
                if (leader) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint64_t hv = desc_sw128_mn(smem_u32(ring + at[h] * SP_SLOT), 8192);
                        const uint32_t p = p0 + (uint32_t) (h * 64);
#pragma unroll
                        for (int k = 0; k < 4; k++) mma_f16_ts(d, p + (k >> 1) * 32 + (k & 1) * 8, hv + k * (2048 >> 4), idesc_v, 1u);
                        mma_commit(&ctl->empty[at[h]]);
                    }
                    mma_commit(&ctl->o_full[buf]);
                }
                __syncwarp();
            }
            __syncwarp();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SP_REGS_SM));
        const int quad = warp & 3, part = (warp - 4) >> 2, row = quad * 32 + lane;
        const int qi = row < rows ? q0 + row / P.gqa : -1;                       // the row's position; -1: sees nothing
        const int lo_q = qi >= 0 ? attn_first_visible(a, qi) : 0;
        const int h = kvh * P.gqa + (row < rows ? row % P.gqa : 0);
        const uint32_t mine = tmem + ((uint32_t) (quad * 32) << 16);
        constexpr float LOG2E = 1.4426950408889634f;
        const float qs = CAP ? ctl->q_scale[row] * a.scale / a.softcap : ctl->q_scale[row] * a.scale, cap = a.softcap;
        const int all_from = attn_first_visible(a, q0 + toks - 1), all_to = q0;   // positions in [all_from, all_to] are visible to every row
        float o[64], m = -INFINITY, l = 0.f, corr1 = 0.f, f1 = 0.f;
        bool bad = false;
#pragma unroll
        for (int i = 0; i < 64; i++) o[i] = 0.f;
        auto add_tile = [&](int j, float corr, float f) {                        // o = o * corr + f * (tile j's weighted sum)
            mbar_wait(&ctl->o_full[j & 1], (uint32_t) ((j / 2) & 1), cta_abort, P.abort_flag);
            __syncwarp();
            fence_after();
            uint32_t v[32];
            if (part < nv) {
                const uint32_t at = mine + O0 + (uint32_t) ((j & 1) * 128 + part * 64);
#pragma unroll
                for (int c = 0; c < 64; c += 32) {
                    TMEM_LD32(at + c, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i++) o[c + i] = fmaf(o[c + i], corr, __uint_as_float(v[i]) * f);
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl->o_free[j & 1]);
        };
        for (int j = 0; j < nt; j++) {   // to the end also after an abort (waits return at once then): the warps meet at a barrier in every round
            const int buf = j & 1, k0 = tile_of(j) * SP_KEYS + part * 64;
            const float * sc = scales + buf * (SP_SCALES / 4) + part * 64;
            mbar_wait(&ctl->sc_full[buf], (uint32_t) ((j / 2) & 1), cta_abort, P.abort_flag);
            mbar_wait(&ctl->s_full[buf], (uint32_t) ((j / 2) & 1), cta_abort, P.abort_flag);
            __syncwarp();
            fence_after();
            float t[64];
            uint32_t * v = reinterpret_cast<uint32_t *>(t);
            const uint32_t at = mine + (uint32_t) (buf * 128 + part * 64);
            TMEM_LD32(at, v);
            TMEM_LD32(at + 32, v + 32);
            tmem_wait_ld();
            // every row sees the whole tile, and its values lie within 2^12 of one another: their scales relative to the tile's largest go into the
            // weights as they are.  Else a row's scales follow the largest product weight x power of two among the positions that it sees
            const float * tail = scales + buf * (SP_SCALES / 4) + 3 * SP_KEYS;
            const int tile0 = tile_of(j) * SP_KEYS;
            const bool whole = tile0 >= all_from && tile0 + SP_KEYS - 1 <= all_to, plain = whole && tail[1] == 0.f;
            float tm = -INFINITY, tw = -INFINITY;
            // two copies: with the test beside it every score of every tile paid for it (3600 instead of 1100 clocks a tile)
            auto take = [&](auto sees) {
#pragma unroll
                for (int i = 0; i < 64; i += 4) {
                    const float4 s4 = *reinterpret_cast<const float4 *>(sc + i);
                    const float f[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        float x = t[i + q] * f[q] * qs;
                        if constexpr (CAP) x = cap * tanhf(x);
                        if (!sees(i + q)) x = -INFINITY;
                        t[i + q] = x;
                        tm = fmaxf(tm, x);
                    }
                }
            };
            if (whole) {
                take([](int) { return true; });
            } else {
                const uint64_t seen = below(qi + 1 - k0) & (~below(lo_q - k0) | below(a.keep_first - k0));
                const uint32_t seen2[2] = {(uint32_t) seen, (uint32_t) (seen >> 32)};
                take([&](int i) { return (seen2[i >> 5] >> (i & 31) & 1u) != 0u; });
            }
            if (!plain) {
#pragma unroll
                for (int i = 0; i < 64; i += 4) {
                    const float4 w4 = *reinterpret_cast<const float4 *>(sc + 2 * SP_KEYS + i);
                    tw = fmaxf(fmaxf(fmaxf(tw, fmaf(t[i], LOG2E, w4.x)), fmaxf(fmaf(t[i + 1], LOG2E, w4.y), fmaf(t[i + 2], LOG2E, w4.z))), fmaf(t[i + 3], LOG2E, w4.w));
                }
            }
            ctl->row_max[buf][part][row] = make_float2(tm, tw);
            asm volatile("bar.sync 1, %0;" ::"n"(SP_SM_THREADS) : "memory");
            const float2 other = ctl->row_max[buf][part ^ 1][row];
            // the exponentials are powers of two, references whole numbers: what joins tiles is exact
            const float here = ceilf(fmaxf(tm, other.x) * LOG2E), mn = fmaxf(m, here), ref = here == -INFINITY ? 0.f : here;
            const float corr = pow2_down(m - mn), part_f = pow2_down(here - mn);
            int top = 0;
            float e4[4] = {0.f, 0.f, 0.f, 0.f}, sum = 0.f;
            if (!plain) {   // the exponents of the weights' own sum, then those of the products weight x power of two in their place
                top = max(__float2int_ru(fmaxf(tw, other.y) - ref), -99);
                const float lift = (float) (14 - top);
#pragma unroll
                for (int i = 0; i < 64; i += 4) {
                    const float4 w4 = *reinterpret_cast<const float4 *>(sc + 2 * SP_KEYS + i);
                    const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float y = fmaf(t[i + q], LOG2E, -ref);
                        e4[q] += ex2(y);
                        t[i + q] = y + (w[q] + lift);
                    }
                }
                sum = (e4[0] + e4[1]) + (e4[2] + e4[3]);
            }
            const float * ratio = plain ? sc + SP_KEYS : ctl->ones;
            const float slope = plain ? LOG2E : 1.f, offset = plain ? -ref : 0.f;
#pragma unroll
            for (int c = 0; c < 64; c += 32) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 r4 = *reinterpret_cast<const float4 *>(ratio + c + i);
                    const float r[4] = {r4.x, r4.y, r4.z, r4.w};
                    float p[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        p[q] = ex2(fmaf(t[c + i + q], slope, offset));
                        e4[q] += p[q];
                        p[q] *= fabsf(r[q]);
                    }
                    split2(p[0], p[1], hi[i / 2], lo[i / 2]);
                    split2(p[2], p[3], hi[i / 2 + 1], lo[i / 2 + 1]);
                }
                TMEM_ST16(at + c, hi);
                TMEM_ST16(at + c + 16, lo);
            }
            if (plain) sum = (e4[0] + e4[1]) + (e4[2] + e4[3]);
            tmem_wait_st();
            const float f = (plain ? tail[2] : __uint_as_float((uint32_t) (top + 100) << 23)) * part_f;   // of the sums: 2^(top - 14 - 13)
            bad = bad || tail[0] != 0.f;
            loads_done(__float_as_uint(f) + (bad ? 1u : 0u));   // both are first used in the next round, when the scales may be another tile's
            fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&ctl->p_full[buf]); mbar_arrive(&ctl->sc_empty[buf]); }
            l = l * corr + sum * part_f;
            m = mn;
            if (j > 0) add_tile(j - 1, corr1, f1);
            corr1 = corr;
            f1 = f;
        }
        add_tile(nt - 1, corr1, f1);
        ctl->row_l[part][row] = l;
        asm volatile("bar.sync 1, %0;" ::"n"(SP_SM_THREADS) : "memory");
        l = ctl->row_l[0][row] + ctl->row_l[1][row];
        if (a.sink && m != -INFINITY) l += ex2(fmaf(io.sink ? io.sink[h] : 0.f, LOG2E, -m));
        const float inv = l > 0.f ? 1.f / l : 0.f;
        // through the ring's memory (every unit has been used; a row's 16-byte pieces rotated by the row), so that a warp stores whole rows
        float * os = reinterpret_cast<float *>(ring);
        if (part < nv) {
#pragma unroll
            for (int i = 0; i < 16; i++)
                *reinterpret_cast<float4 *>(os + row * 128 + ((part * 16 + i + row) & 31) * 4) = make_float4(o[4 * i] * inv, o[4 * i + 1] * inv, o[4 * i + 2] * inv, o[4 * i + 3] * inv);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(SP_SM_THREADS) : "memory");
        const int DV = a.vdim, w = warp - 4;
        for (int r = w * 16; r < w * 16 + 16 && r < rows; r++) {
            const int64_t tok = t_begin + q0 + r / P.gqa;
            const int hh = kvh * P.gqa + r % P.gqa;
#pragma unroll
            for (int c = 0; c < 128; c += 32) {
                const int d = c + lane;
                if (d < DV) put((OT *) P.out, tok * ((int64_t) a.heads * DV) + (int64_t) hh * DV + d, os[r * 128 + (((d >> 2) + r) & 31) * 4 + (d & 3)] * gate_factor(io, tok, hh, d, DV));
            }
        }
        if (bad) {   // what is no number among the values that a row sees is its result
            __syncwarp();   // over what other lanes have stored
            const uint8_t * tiles = P.ws + ((int64_t) blockIdx.x * P.slots + t_begin / SP_KEYS + e) * sp_tile_bytes(nd, nv);
#pragma unroll 1
            for (int i = lane; i < 16 * DV; i += 32) {
                const int r = w * 16 + i / DV, d = i % DV;
                if (r >= rows) break;
                const int64_t tok = t_begin + q0 + r / P.gqa;
                const int hh = kvh * P.gqa + r % P.gqa;
                const float y = not_numbers(P, tiles, e, kvh, q0 + r / P.gqa, d);
                if (!(fabsf(y) < INFINITY)) put((OT *) P.out, tok * ((int64_t) a.heads * DV) + (int64_t) hh * DV + d, y * gate_factor(io, tok, hh, d, DV));
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

template <typename OT, bool CAP>
int launch_typed(const SplitParams & P, const dim3 & grid, size_t smem, cudaStream_t st) {
    static FuncAttrCache cache;
    const cudaError_t e = ensure_dyn_smem(cache, (const void *) k_attn_split<OT, CAP>, smem, true);
    if (e != cudaSuccess) return (int) e;
    static std::atomic<bool> fits{false};   // the roles' registers are within the launch's: beyond them the softmax warps would wait without end
    if (!fits.load(std::memory_order_relaxed)) {
        cudaFuncAttributes f;
        const cudaError_t ea = cudaFuncGetAttributes(&f, k_attn_split<OT, CAP>);
        if (ea != cudaSuccess) return (int) ea;
        if (f.numRegs * SP_THREADS < 128 * SP_REGS_FEW + SP_SM_THREADS * SP_REGS_SM) return (int) cudaErrorLaunchOutOfResources;
        fits.store(true, std::memory_order_relaxed);
    }
    return launch_dep(k_attn_split<OT, CAP>, grid, dim3(SP_THREADS), smem, st, P);
}
int split_slots(int n_tokens, int n_entries) { return n_tokens / SP_KEYS + n_entries; }   // floor(off / 128) + e are distinct runs of slots

}  // namespace

// Scratch of one kv head; all heads at once up to SP_SCRATCH bytes (2000 tiles of 128-wide heads: far more CTAs than SMs), beyond that in groups.
constexpr size_t SP_SCRATCH = (size_t) 256 << 20;
static bool split_shape(const AttnParams & a) {
    return a.dim > 0 && a.dim <= 64 * SP_MAX_ND && a.vdim > 0 && a.vdim <= 64 * SP_MAX_NV && a.kv_heads > 0 && a.heads % a.kv_heads == 0 && a.heads / a.kv_heads <= 128;
}
static size_t split_head_bytes(const AttnParams & a, int n_tokens, int n_entries) {
    return (size_t) split_slots(n_tokens, n_entries) * (size_t) sp_tile_bytes((a.dim + 63) / 64, (a.vdim + 63) / 64);
}
size_t attn_split_bytes(const AttnParams & a, int n_tokens, int n_entries) {
    if (!split_shape(a)) return 0;
    const size_t head = split_head_bytes(a, n_tokens, n_entries);
    return head * std::min<size_t>((size_t) a.kv_heads, std::max<size_t>(1, SP_SCRATCH / head));
}
bool attn_split_ok(const AttnIO & io, const BatchView & b, const AttnParams & a) {
    if (!io.split_ws || !split_shape(a) || b.n_entries > 65535) return false;
    const int tok_per_cta = 128 / (a.heads / a.kv_heads);
    return (b.max_n - 1) / tok_per_cta < 65535 && attn_split_bytes(a, b.n_tokens, b.n_entries) <= io.split_bytes;   // a grid's second dimension
}
int launch_attn_split(const AttnIO & io, const BatchView & b, const AttnParams & a, void * out, int otype, cudaStream_t st) {
    SplitParams P{};
    P.io = io; P.a = a; P.off = b.off;
    P.ws = (uint8_t *) io.split_ws;
    P.slots = split_slots(b.n_tokens, b.n_entries);
    P.out = out;
    P.nd = (a.dim + 63) / 64; P.nv = (a.vdim + 63) / 64;
    P.gqa = a.heads / a.kv_heads;
    P.tok_per_cta = 128 / P.gqa;
    P.slots_ring = 13 - 2 * P.nd;   // with the queries' 2 nd pieces what an SM's shared memory holds
    P.abort_flag = abort_flag();
    const int group = (int) (attn_split_bytes(a, b.n_tokens, b.n_entries) / split_head_bytes(a, b.n_tokens, b.n_entries));
    const size_t smem = 1024 + (size_t) P.nd * 32768 + (size_t) P.slots_ring * SP_SLOT + 2 * SP_SCALES + sizeof(SpCtl);
    for (P.kv_first = 0; P.kv_first < a.kv_heads; P.kv_first += group) {
        const unsigned heads = (unsigned) std::min(group, a.kv_heads - P.kv_first);
        g_launches += 2;
        int rc = launch_dep(k_split_kv, dim3((unsigned) ((b.max_n + SP_KEYS - 1) / SP_KEYS), heads, (unsigned) b.n_entries), dim3(256), 0, st, P);
        if (rc) return rc;
        const dim3 grid(heads, (unsigned) ((b.max_n + P.tok_per_cta - 1) / P.tok_per_cta), (unsigned) b.n_entries);
        if (otype == T_BF16) rc = a.softcap > 0.f ? launch_typed<__nv_bfloat16, true>(P, grid, smem, st) : launch_typed<__nv_bfloat16, false>(P, grid, smem, st);
        else rc = a.softcap > 0.f ? launch_typed<float, true>(P, grid, smem, st) : launch_typed<float, false>(P, grid, smem, st);
        if (rc) return rc;
    }
    return 0;
}

}  // namespace pb
