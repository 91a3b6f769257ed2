// prima.cpp_b200/csrc/attn_tc.cu — prompt attention over the f16 cache on the 5th-generation tensor cores (k_attn_prefill_tc): the FA-off chain of the
// reference's graph (ggml-cuda.cu:1737-1881; CPU ggml.c:12377-12600, 13783-13880): q rounded to f16, scores in fp32, softmax over the
// row, probabilities rounded to f16 AFTER they are normalised, values weighed in fp32.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "launch.h"
#include "tc.cuh"

namespace pb {
namespace {

// One CTA: 128 query rows (the heads of a GQA group x 128 / group consecutive tokens) of one kv head, so that a key tile serves the whole group
// and the causal edge costs one tile.  The rounding of normalised probabilities needs the row's maximum and sum first, hence two
// walks over the keys: the first takes S = Q K^T for the maximum and the sum; the second goes back from the last tile (whose S is still
// there), takes S again, writes P = f16(exp(S - max) / sum) over it in tensor memory and adds P V.  A row's result does not depend on what
// else is in the launch: a tile that it does not see adds zeros.
// Tensor memory: 256 columns, S / P | second S in the first walk, O in the second one; with 104 KB of shared memory two CTAs share an SM, and
// one's softmax lies beside the other's MMAs, start and end.
//   warp 0       TMA: key and value tiles of 128 positions (two boxes of 64 head entries each), ring of AT_STAGES
//   warp 1       MMA issuer, owner of the tensor memory
//   warps 2 - 9  softmax: thread = (row, half of the tile's keys, 32 at a time); row = TMEM lane
// Bound: 2 exponentials per score on the MUFU (16 a clock: 2048 clocks a 128 x 128 tile) against 1536 clocks of MMA; two CTAs together take
// 1100 clocks a tile in the first walk and 1550 in the second, a CTA's start and end 6500.  Measured at 2048 tokens, 32 heads over 8:
// 2994 us with the scores in shared memory and fp32 FMA before, 80.6 us (427 TFLOP/s of visible pairs; 85 with launch and wait); one CTA to an SM with both
// operands twice in tensor memory took 101 us.  512 tokens: 120 -> 17.5 us; 16 tokens behind 2000: 201 -> 47 us.  A first prompt of 16 / 32 / 64 tokens
// (32 heads over 8), which is a start and an end and little between: 5.9 / 6.6 / 10.0 -> 7.4 / 8.1 / 8.7 us.
constexpr int AT_STAGES = 2, AT_STAGE = 32768, AT_BLOCK = 16384;
constexpr int AT_PARTS = 2, AT_COLS = 128 / AT_PARTS, AT_SM_THREADS = 128 * AT_PARTS, AT_THREADS = 64 + AT_SM_THREADS;

struct AtCtl {
    uint64_t full[AT_STAGES], empty[AT_STAGES], s_full[2], s_free[2], p_full, o_full;
    uint32_t tmem_base;
    int abort, bad_any;
    int lim_min[4], lim_max[4];
    int first_bad[128];        // per value column: first position with a non-finite value that some row of the tile does not see
    float row_m[AT_PARTS][128];
    double row_l[AT_PARTS][128];
};
struct AtParams {
    const float * q; float * out; const int32_t * pos;
    int n_head, gqa, tok_per_cta, n_tok;
    float c;                   // scale * log2(e)
    int * abort_flag;
};

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void softmax_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(AT_SM_THREADS) : "memory"); }

// first entry of row r of the tile that starts at token t0: token t0 + r / gqa, head r % gqa of the group (a division costs more than a row's walk over
// the next 16: the callers count on)
__device__ __forceinline__ int64_t row_offset(const AtParams & P, int t0, int hk, int r) {
    return ((int64_t) (t0 + r / P.gqa) * P.n_head + hk * P.gqa + r % P.gqa) * 128;
}
__global__ void __launch_bounds__(AT_THREADS, 2)
    k_attn_prefill_tc(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ AtParams P) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t * q_s = smem, * ring = smem + AT_STAGE;                        // queries: two blocks of 128 rows x 64 entries
    AtCtl * ctl = reinterpret_cast<AtCtl *>(ring + AT_STAGES * AT_STAGE);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int hk = blockIdx.x, t0 = ((int) gridDim.y - 1 - (int) blockIdx.y) * P.tok_per_cta;   // long rows first
    const int rows = min(P.tok_per_cta, P.n_tok - t0) * P.gqa;
    volatile int * cta_abort = &ctl->abort;
    int u = 0;                                                             // tiles loaded (warp 0) or used (warp 1)
    auto load = [&](const CUtensorMap * m, int tile) {
        const int s = u % AT_STAGES;
        if (u >= AT_STAGES) mbar_wait(&ctl->empty[s], (uint32_t) ((u / AT_STAGES - 1) & 1), cta_abort, P.abort_flag);
        __syncwarp();
        if (elect_one()) {
            const uint32_t dst = smem_u32(ring + s * AT_STAGE), bar = smem_u32(&ctl->full[s]);
            mbar_arrive_expect_tx(&ctl->full[s], AT_STAGE);
            tma_load<1>(dst, m, hk * 128, tile * 128, 0, bar);
            tma_load<1>(dst + AT_BLOCK, m, hk * 128 + 64, tile * 128, 0, bar);
        }
        __syncwarp();
        u++;
    };
    int lim = -1;                                                          // softmax threads: the last position their row sees
    if (warp == 0) {
        if (lane == 0) {
            prefetch_map(&map_k);
            prefetch_map(&map_v);
            for (int i = 0; i < AT_STAGES; i++) { mbar_init(&ctl->full[i], 1); mbar_init(&ctl->empty[i], 1); }
            for (int i = 0; i < 2; i++) { mbar_init(&ctl->s_full[i], 1); mbar_init(&ctl->s_free[i], 4 * AT_PARTS); }
            mbar_init(&ctl->p_full, 4 * AT_PARTS);
            mbar_init(&ctl->o_full, 1);
            ctl->abort = 0; ctl->bad_any = 0;
            mbar_fence_init();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
        load(&map_k, 0);                                                   // on its way while the queries are fetched
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        for (int i = lane; i < 128; i += 32) ctl->first_bad[i] = 0x7fffffff;
    } else {
        // queries -> f16 in the swizzle-128B image: a warp reads whole rows (a lane: four entries), 16 of them in flight; rows beyond the tile are zero
        const int w = warp - 2;
        const float * src = P.q + row_offset(P, t0, hk, w * 16) + 4 * lane;
        int rem = w * 16 % P.gqa;
        float4 a[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            a[i] = w * 16 + i < rows ? *reinterpret_cast<const float4 *>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
            src += 128;
            if (++rem == P.gqa) { rem = 0; src += (P.n_head - P.gqa) * 128; }
        }
        const int trow = (warp & 3) * 32 + lane;
        if (trow < rows) lim = max(P.pos[t0 + trow / P.gqa], -1);
        const int lo = __reduce_min_sync(0xffffffffu, trow < rows ? lim : 0x7fffffff), hi = __reduce_max_sync(0xffffffffu, lim);
        if (lane == 0) { ctl->lim_min[warp & 3] = lo; ctl->lim_max[warp & 3] = hi; }
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int row = w * 16 + i;
            *reinterpret_cast<uint2 *>(q_s + (lane >> 4) * AT_BLOCK + (row >> 3) * 1024 + (row & 7) * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4) + (lane & 1) * 8) =
                make_uint2(pack_f16(a[i].x, a[i].y), pack_f16(a[i].z, a[i].w));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *(volatile uint32_t *) &ctl->tmem_base;
    const int lim_min = min(min(ctl->lim_min[0], ctl->lim_min[1]), min(ctl->lim_min[2], ctl->lim_min[3]));   // positions up to it every row sees,
    const int lim_max = max(max(ctl->lim_max[0], ctl->lim_max[1]), max(ctl->lim_max[2], ctl->lim_max[3]));   // beyond this one none
    const int n = (lim_max + 128) >> 7;                                    // key tiles
    constexpr uint32_t S0 = 0, O0 = 128;

    if (warp == 0) {
        for (int j = 1; j < n && !*cta_abort; j++) load(&map_k, j);
        for (int j = n - 1; j >= 0 && !*cta_abort; j--) {                  // V(n - 1) K(n - 2) V(n - 2) ...
            if (j < n - 1) load(&map_k, j);
            load(&map_v, j);
        }
        if (n == 0) mbar_wait(&ctl->full[0], 0u, cta_abort, P.abort_flag);   // no copy outlives the CTA
        __syncwarp();
    } else if (warp == 1) {
        constexpr uint32_t idesc = (1u << 4) | ((uint32_t) (128 >> 3) << 17) | ((uint32_t) (128 >> 4) << 24), idesc_v = idesc | (1u << 16);
        const uint64_t dq = desc_sw128(smem_u32(q_s));
        auto scores = [&](int buf, bool reused, uint32_t phase) {
            const int s = u % AT_STAGES;
            mbar_wait(&ctl->full[s], (uint32_t) ((u / AT_STAGES) & 1), cta_abort, P.abort_flag);
            if (reused) mbar_wait(&ctl->s_free[buf], phase, cta_abort, P.abort_flag);
            __syncwarp();
            fence_after();
            const uint64_t dk = desc_sw128(smem_u32(ring + s * AT_STAGE));
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < 8; k++)
                    mma_f16<1>(tmem + S0 + buf * 128, dq + (k >> 2) * (AT_BLOCK >> 4) + 2 * (k & 3), dk + (k >> 2) * (AT_BLOCK >> 4) + 2 * (k & 3), idesc, (uint32_t) (k != 0));
                mma_commit(&ctl->empty[s]);
                mma_commit(&ctl->s_full[buf]);
            }
            __syncwarp();
            u++;
        };
        for (int j = 0; j < n && !*cta_abort; j++) scores((n - 1 - j) & 1, j >= 2, (uint32_t) ((j / 2 - 1) & 1));   // the last tile in the first columns
        for (int j = n - 1, i = 0; j >= 0 && !*cta_abort; j--, i++) {
            if (i > 0) scores(0, false, 0);
            const int s = u % AT_STAGES;
            mbar_wait(&ctl->full[s], (uint32_t) ((u / AT_STAGES) & 1), cta_abort, P.abort_flag);
            mbar_wait(&ctl->p_full, (uint32_t) (i & 1), cta_abort, P.abort_flag);
            __syncwarp();
            fence_after();
            const uint64_t dv = desc_sw128_mn(smem_u32(ring + s * AT_STAGE), AT_BLOCK);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < 8; k++) mma_f16_ts(tmem + O0, tmem + S0 + (k >> 2) * 64 + (k & 3) * 8, dv + k * (2048 >> 4), idesc_v, (uint32_t) ((i | k) != 0));
                mma_commit(&ctl->empty[s]);
                if (j == 0) mma_commit(&ctl->o_full);
            }
            __syncwarp();
            u++;
        }
        __syncwarp();
    } else {
        const int quad = warp & 3, part = (warp - 2) >> 2, row = quad * 32 + lane, tid = threadIdx.x - 64;
        const uint32_t mine = tmem + ((uint32_t) (quad * 32) << 16) + (uint32_t) (part * AT_COLS);   // this thread's row and columns of S
        const float c = P.c;
        float t[32];
        // 32 scores from position k0 on, times scale * log2(e); a masked score is -inf
        auto take = [&](uint32_t addr, int k0) {
            uint32_t * v = reinterpret_cast<uint32_t *>(t);
            TMEM_LD32(addr, v);
            tmem_wait_ld();
            if (k0 + 31 <= lim_min) {
#pragma unroll
                for (int i = 0; i < 32; i++) t[i] *= c;
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) t[i] = k0 + i <= lim ? t[i] * c : -INFINITY;
            }
        };
        float m = -INFINITY;
        double l = 0.0;
        uint32_t ph[2] = {0u, 0u};
        for (int j = 0; j < n && !*cta_abort; j++) {
            const int buf = (n - 1 - j) & 1;
            mbar_wait(&ctl->s_full[buf], buf ? ph[1] : ph[0], cta_abort, P.abort_flag);
            if (buf) ph[1] ^= 1u; else ph[0] ^= 1u;
            __syncwarp();
            fence_after();
#pragma unroll
            for (int h = 0; h < AT_COLS; h += 32) {
                const bool some = j * 128 + part * AT_COLS + h <= lim_max;   // else nothing of these 32 positions is visible to any row
                if (some) take(mine + S0 + (uint32_t) (buf * 128 + h), j * 128 + part * AT_COLS + h);
                if (h + 32 == AT_COLS) {
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctl->s_free[buf]);
                }
                if (!some) continue;
                float tm[4] = {t[0], t[1], t[2], t[3]};
#pragma unroll
                for (int i = 4; i < 32; i++) tm[i & 3] = fmaxf(tm[i & 3], t[i]);
                const float mn = fmaxf(fmaxf(m, fmaxf(tm[0], tm[1])), fmaxf(tm[2], tm[3]));
                if (mn == -INFINITY) {   // nothing visible yet (a NaN is no maximum: it has to reach the sum)
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (t[i] != t[i]) l = (double) t[i];
                } else {
                    float e[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int i = 0; i < 32; i++) e[i & 3] += ex2(t[i] - mn);
                    l = l * (double) ex2(m - mn) + (double) ((e[0] + e[1]) + (e[2] + e[3]));
                    m = mn;
                }
            }
        }
        ctl->row_m[part][row] = m;
        ctl->row_l[part][row] = l;
        softmax_barrier();
        m = -INFINITY;
#pragma unroll
        for (int i = 0; i < AT_PARTS; i++) m = fmaxf(m, ctl->row_m[i][row]);
        l = 0.0;
#pragma unroll
        for (int i = 0; i < AT_PARTS; i++) {
            const float mi = ctl->row_m[i][row];
            l += mi == -INFINITY ? ctl->row_l[i][row] : ctl->row_l[i][row] * (double) ex2(mi - m);
        }
        const float inv = lim >= 0 ? (float) (1.0 / l) : 0.f;
        if (lim < 0) m = 0.f;
        for (int j = n - 1, i2 = 0; j >= 0 && !*cta_abort; j--, i2++) {
            if (i2 > 0) {
                mbar_wait(&ctl->s_full[0], ph[0], cta_abort, P.abort_flag);
                ph[0] ^= 1u;
                __syncwarp();
            }
            fence_after();
#pragma unroll
            for (int h = 0; h < AT_COLS; h += 32) {   // P goes over the first 32 of this thread's own columns, which have been read by then
                const int k0 = j * 128 + part * AT_COLS + h;
                uint32_t p[16];
                if (k0 <= lim_max) take(mine + S0 + (uint32_t) h, k0);
                if (k0 > lim_max) {
#pragma unroll
                    for (int i = 0; i < 16; i++) p[i] = 0u;
                } else if (k0 + 31 <= lim_min) {
#pragma unroll
                    for (int i = 0; i < 16; i++) p[i] = pack_f16(ex2(t[2 * i] - m) * inv, ex2(t[2 * i + 1] - m) * inv);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const float a = k0 + 2 * i <= lim ? ex2(t[2 * i] - m) * inv : 0.f, b = k0 + 2 * i + 1 <= lim ? ex2(t[2 * i + 1] - m) * inv : 0.f;
                        p[i] = pack_f16(a, b);
                    }
                }
                TMEM_ST16(mine + S0 + (uint32_t) (h / 2), p);
            }
            tmem_wait_st();
            if (j * 128 + 127 > lim_min) {
                // the tile holds positions that some row does not see.  A weight of zero does not silence a value that is no number: positions no row
                // sees are cleared (the cache may hold anything there), non-finite values that only later rows see are taken out and remembered
                const int uv = n + 2 * i2, s = uv % AT_STAGES;
                mbar_wait(&ctl->full[s], (uint32_t) ((uv / AT_STAGES) & 1), cta_abort, P.abort_flag);
                const int key = tid >> 1, kp = j * 128 + key, blk = tid & 1;
                uint8_t * vr = ring + s * AT_STAGE + blk * AT_BLOCK + key * 128;
                if (kp > lim_max) {
#pragma unroll
                    for (int i = 0; i < 8; i++) *reinterpret_cast<uint4 *>(vr + 16 * ((i + key) & 7)) = make_uint4(0u, 0u, 0u, 0u);
                } else if (kp > lim_min) {
#pragma unroll
                    for (int c8 = 0; c8 < 8; c8++) {   // in another order for every row: the same piece of all rows lies in the same banks
                        const int ch = (c8 + key) & 7;
                        const uint4 w = *reinterpret_cast<const uint4 *>(vr + 16 * ch);
                        const uint32_t x[4] = {w.x, w.y, w.z, w.w};
                        bool any = false;
#pragma unroll
                        for (int i = 0; i < 4; i++) any = any || (x[i] & 0x7c00u) == 0x7c00u || (x[i] & 0x7c000000u) == 0x7c000000u;
                        if (any) {
                            uint16_t * hv = reinterpret_cast<uint16_t *>(vr + 16 * ch);
#pragma unroll 1
                            for (int i = 0; i < 8; i++)
                                if ((hv[i] & 0x7c00) == 0x7c00) {
                                    atomicMin(&ctl->first_bad[blk * 64 + ((ch ^ (key & 7)) << 3) + i], kp);
                                    ctl->bad_any = 1;
                                    hv[i] = 0;
                                }
                        }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl->p_full);
        }
        if (n > 0) {
            mbar_wait(&ctl->o_full, 0u, cta_abort, P.abort_flag);
            softmax_barrier();   // every warp has looked through its values
            fence_after();
        } else {
            mbar_wait(&ctl->full[0], 0u, cta_abort, P.abort_flag);   // key tile 0 is on its way into the ring all the same
        }
        // the result goes through the ring's memory (every tile has been used; row r's 16-byte pieces rotated by r) so that a warp stores whole rows
        float * os = reinterpret_cast<float *>(ring);
#pragma unroll
        for (int h = 0; h < AT_COLS; h += 32) {
            if (n > 0) {
                uint32_t * v = reinterpret_cast<uint32_t *>(t);
                TMEM_LD32(mine + O0 + (uint32_t) h, v);
                tmem_wait_ld();
                if (*(volatile int *) &ctl->bad_any) {
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (lim >= ctl->first_bad[part * AT_COLS + h + i]) t[i] = __int_as_float(0x7fc00000);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) t[i] = 0.f;
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
                *reinterpret_cast<float4 *>(os + row * 128 + (((part * AT_COLS + h) / 4 + i + row) & 31) * 4) = make_float4(t[4 * i], t[4 * i + 1], t[4 * i + 2], t[4 * i + 3]);
        }
        softmax_barrier();
        const int r0 = (warp - 2) * 16;
        float * out = P.out + row_offset(P, t0, hk, r0) + 4 * lane;
        int rem = r0 % P.gqa;
#pragma unroll
        for (int i0 = 0; i0 < 16; i0 += 8) {
            float4 x[8];
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = *reinterpret_cast<const float4 *>(os + (r0 + i0 + i) * 128 + ((lane + r0 + i0 + i) & 31) * 4);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (r0 + i0 + i < rows) *reinterpret_cast<float4 *>(out) = x[i];
                out += 128;
                if (++rem == P.gqa) { rem = 0; out += (P.n_head - P.gqa) * 128; }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
    }
}

}  // namespace

bool attn_prefill_tc_ok(const float * q, const __half * kcache, const __half * vcache, const float * out, int n_head, int n_head_kv, int D, int n_kv_max) {
    const uintptr_t a = (uintptr_t) q | (uintptr_t) kcache | (uintptr_t) vcache | (uintptr_t) out;
    return D == 128 && n_head_kv > 0 && n_head % n_head_kv == 0 && n_head / n_head_kv <= 128 && n_kv_max > 0 && (a & 15) == 0;
}

int launch_attn_prefill_tc(const float * q, const __half * kcache, const __half * vcache, float * out, int n_head, int n_head_kv, const int32_t * pos_dev, int n_tok,
                           int n_kv_max, float scale, cudaStream_t st) {
    constexpr size_t smem = 1024 + (size_t) (AT_STAGES + 1) * AT_STAGE + sizeof(AtCtl);
    static_assert(smem <= 232448, "shared memory of an SM");
    static FuncAttrCache cache;
    const cudaError_t e = ensure_dyn_smem(cache, (const void *) k_attn_prefill_tc, smem, true);
    if (e != cudaSuccess) return (int) e;
    const int gqa = n_head / n_head_kv;
    const AtParams P{q, out, pos_dev, n_head, gqa, 128 / gqa, n_tok, scale * 1.4426950408889634f, abort_flag()};
    const int64_t ld = (int64_t) n_head_kv * 128;
    CUtensorMap mk, mv;
    int rc = make_map(mk, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, kcache, ld, n_kv_max, 1, ld, 0, 128);
    if (!rc) rc = make_map(mv, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, vcache, ld, n_kv_max, 1, ld, 0, 128);
    if (rc) return rc;
    const dim3 grid((unsigned) n_head_kv, (unsigned) ((n_tok + P.tok_per_cta - 1) / P.tok_per_cta));
    k_attn_prefill_tc<<<grid, AT_THREADS, smem, st>>>(mk, mv, P);
    return (int) cudaGetLastError();
}

}  // namespace pb
