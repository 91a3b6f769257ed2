// prima.cpp_b200/csrc/attn_tc.cu — prompt attention over the f16 cache on the 5th-generation tensor cores (k_attn_prefill_tc): the FA-off chain of the
// reference's graph (ggml-cuda.cu:1737-1881; CPU ggml.c:12377-12600, 13783-13880): q rounded to f16, scores in fp32, softmax over the
// row, values weighed in fp32.  Probabilities are rounded to f16 as there, of rows of 160 positions and more in front of the division by the row's sum: the
// rounding is the same share of a weight, and fewer weights fall below f16's normal range.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>

#include "launch.h"
#include "tc.cuh"

namespace pb {
namespace {

// An item: 128 query rows (the heads of a GQA group x 128 / group consecutive tokens) of one kv head, so that a key tile serves the whole group
// and the causal edge costs one tile.  One walk over the keys: S = Q K^T, weights P = f16(exp(S - reference)) over S in tensor memory, O += P V, divided by the row's
// sum at the end.  A row's reference is the largest score of its first tile; a later tile is weighed by it at once, and only where a score turns out to lie beyond it by
// more than 2^8 the row's sum and O are scaled to the new one and the tile is weighed again (each row by its own scores: a row's result does not
// depend on what else is in the launch; a tile that it does not see adds zeros).
// Tensor memory: 256 columns, S / P | O; with 104 KB of shared memory two CTAs share an SM, and one's softmax lies beside the other's MMAs, start and end.
//   warp 0       TMA: key and value tiles of 128 positions (two boxes of 64 head entries each), ring of AT_STAGES
//   warp 1       MMA issuer, owner of the tensor memory
//   warps 2 - 9  softmax: thread = (row, half of the tile's keys, 32 at a time); row = TMEM lane
// At most two CTAs to an SM, which take items in turns: a CTA that ends is replaced only once its neighbour on the SM has ended, too (measured: slots stayed
// empty for 10 us), and the start of a CTA costs 1 us.
// Bound: a tile's chain of about 3500 clocks (S after P 1300, weights 1450 .. 1700, agreement on the row's score 230, stores and barriers 200), of which two CTAs hide
// half of each other's, and 5 us per item for queries, last P V and output.  1024 clocks a tile are the MUFU's, 1450 the MMAs'.
// us in a row of calls, two walks (all scores twice, for maximum and sum first) and an item a CTA / this: 32 heads over 8, 2048 tokens 80.4 / 52.5 (654 TFLOP/s of
// visible pairs), 700 23.9 / 19, 512 17.8 / 13.6, 300 13.9 / 11.6, 250 11.8 / 11.4, 128 9.6 / 9.0, 16 7.8 / 7.1, 16 behind 2000 49 / 35; 8 heads over 4, 1500 behind
// 548 51 / 37.  One walk with an item a CTA took 58.6 at 2048; the maximum in a pass of its own over S in every tile 50.9, but 37 for 16 behind 2000 and 39 for 1500
// behind 548; weights as two f16 numbers, which need no look at short rows and are within 1.4e-6 of 64 bits, 61.5.  Error against 64 bits at 2048 tokens 2.02e-4 / 1.99e-4.
constexpr int AT_STAGES = 2, AT_STAGE = 32768, AT_BLOCK = 16384;
// Rows that see fewer positions have their weights normalised before they are rounded, as the reference does: with few weights the two roundings differ by more
// than 2e-5 of values around 1 (2.3e-5 at 121 positions, falling with the root of their number).  The tiles such rows end in are looked at first.
constexpr int AT_EXACT = 160;
constexpr int AT_PARTS = 2, AT_COLS = 128 / AT_PARTS, AT_SM_THREADS = 128 * AT_PARTS, AT_THREADS = 64 + AT_SM_THREADS;

struct AtCtl {
    uint64_t full[AT_STAGES], empty[AT_STAGES], s_full, s_free, p_full, o_full;
    uint32_t tmem_base;
    int abort, bad_any;
    int lim_min[4], lim_max[4];
    int first_bad[128];        // per value column: first position with a non-finite value that some row of the tile does not see
    float row_m[2][AT_PARTS][128];   // by tile parity
    double row_l[AT_PARTS][128];
};
struct AtParams {
    const float * q; float * out; const int32_t * pos;
    int n_head, n_head_kv, gqa, tok_per_cta, n_tok, items;   // items: kv heads x tiles of tok_per_cta tokens
    float c, sign;             // |scale| * log2(e); the scale's sign goes to the queries
    int * abort_flag;
};

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// the two warps that hold the same rows
__device__ __forceinline__ void rows_barrier(int quad) { asm volatile("bar.sync %0, %1;" ::"r"(2 + quad), "n"(32 * AT_PARTS) : "memory"); }
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
    volatile int * cta_abort = &ctl->abort;
    int u = 0;                                                             // tiles loaded (warp 0) or used (warp 1)
    if (warp == 0 && lane == 0) {
        prefetch_map(&map_k);
        prefetch_map(&map_v);
        for (int i = 0; i < AT_STAGES; i++) { mbar_init(&ctl->full[i], 1); mbar_init(&ctl->empty[i], 1); }
        mbar_init(&ctl->s_full, 1);
        mbar_init(&ctl->s_free, 4 * AT_PARTS);
        mbar_init(&ctl->p_full, 4 * AT_PARTS);
        mbar_init(&ctl->o_full, 1);
        ctl->abort = 0;
        mbar_fence_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        pdl_trigger();   // behind the allocation: a later kernel's CTA on this SM must not take the columns first and wait for this one
    }
    pdl_wait();                                                            // queries, positions, keys and values may be the kernel in front's
    uint32_t tmem = 0, tiles = 0, looks = 0, loads = 0, o_phase = 0;       // of the items in front: key tiles, tiles looked at, loads
    for (int round = 0;; round++) {
        // items by falling length for a prompt: there and back again over the CTAs evens them out
        const int item = round * (int) gridDim.x + ((round & 1) ? (int) gridDim.x - 1 - (int) blockIdx.x : (int) blockIdx.x);
        if (item >= P.items) break;
        const int hk = item % P.n_head_kv, t0 = ((P.items - 1 - item) / P.n_head_kv) * P.tok_per_cta;
        const int rows = min(P.tok_per_cta, P.n_tok - t0) * P.gqa;
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
            __syncwarp();
            load(&map_k, 0);                                                   // on its way while the queries are fetched
        } else if (warp == 1) {
            for (int i = lane; i < 128; i += 32) ctl->first_bad[i] = 0x7fffffff;
            if (lane == 0) ctl->bad_any = 0;
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
                    make_uint2(pack_f16(a[i].x * P.sign, a[i].y * P.sign), pack_f16(a[i].z * P.sign, a[i].w * P.sign));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        fence_before();
        __syncthreads();
        fence_after();
        tmem = *(volatile uint32_t *) &ctl->tmem_base;
        const int lim_min = min(min(ctl->lim_min[0], ctl->lim_min[1]), min(ctl->lim_min[2], ctl->lim_min[3]));   // positions up to it every row sees,
        const int lim_max = max(max(ctl->lim_max[0], ctl->lim_max[1]), max(ctl->lim_max[2], ctl->lim_max[3]));   // beyond this one none
        const int n = (lim_max + 128) >> 7;                                    // key tiles
        const int look = lim_min < AT_EXACT ? min(n, (AT_EXACT + 127) / 128) : 0;      // tiles looked at first, for the maximum and the sum of rows that end in them
        constexpr uint32_t S0 = 0, O0 = 128;

        if (warp == 0) {
            for (int j = 1; j < look; j++) load(&map_k, j);
            for (int j = 0; j < n && !*cta_abort; j++) {                       // K(0) V(0) K(1) V(1) ...
                if (j > 0 || look > 0) load(&map_k, j);
                load(&map_v, j);
            }
            __syncwarp();
        } else if (warp == 1) {
            constexpr uint32_t idesc = (1u << 4) | ((uint32_t) (128 >> 3) << 17) | ((uint32_t) (128 >> 4) << 24), idesc_v = idesc | (1u << 16);
            const uint64_t dq = desc_sw128(smem_u32(q_s));
            auto scores = [&] {                                                // behind the P V that reads this tensor memory: MMAs run in order
                const int s = u % AT_STAGES;
                mbar_wait(&ctl->full[s], (uint32_t) ((u / AT_STAGES) & 1), cta_abort, P.abort_flag);
                __syncwarp();
                fence_after();
                const uint64_t dk = desc_sw128(smem_u32(ring + s * AT_STAGE));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        mma_f16<1>(tmem + S0, dq + (k >> 2) * (AT_BLOCK >> 4) + 2 * (k & 3), dk + (k >> 2) * (AT_BLOCK >> 4) + 2 * (k & 3), idesc, (uint32_t) (k != 0));
                    mma_commit(&ctl->empty[s]);
                    mma_commit(&ctl->s_full);
                }
                __syncwarp();
                u++;
            };
            for (int j = 0; j < look; j++) {
                scores();
                mbar_wait(&ctl->s_free, (looks + (uint32_t) j) & 1, cta_abort, P.abort_flag);
            }
            for (int j = 0; j < n && !*cta_abort; j++) {
                scores();
                const int s = u % AT_STAGES;
                mbar_wait(&ctl->full[s], (uint32_t) ((u / AT_STAGES) & 1), cta_abort, P.abort_flag);
                mbar_wait(&ctl->p_full, (tiles + (uint32_t) j) & 1, cta_abort, P.abort_flag);
                __syncwarp();
                fence_after();
                const uint64_t dv = desc_sw128_mn(smem_u32(ring + s * AT_STAGE), AT_BLOCK);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 8; k++) mma_f16_ts(tmem + O0, tmem + S0 + (k >> 2) * 64 + (k & 3) * 8, dv + k * (2048 >> 4), idesc_v, (uint32_t) ((j | k) != 0));
                    mma_commit(&ctl->empty[s]);
                    if (j == n - 1) mma_commit(&ctl->o_full);
                }
                __syncwarp();
                u++;
            }
            if (n == 0) {   // no row sees anything: key tile 0, which was loaded all the same, is handed back
                const int s = u % AT_STAGES;
                mbar_wait(&ctl->full[s], (uint32_t) ((u / AT_STAGES) & 1), cta_abort, P.abort_flag);
                __syncwarp();
                if (elect_one()) mbar_arrive(&ctl->empty[s]);
                u++;
            }
            __syncwarp();
        } else {
            const int quad = warp & 3, part = (warp - 2) >> 2, row = quad * 32 + lane, tid = threadIdx.x - 64;
            const uint32_t mine = tmem + ((uint32_t) (quad * 32) << 16) + (uint32_t) (part * AT_COLS);   // this thread's row and columns of S
            const float c = P.c;
            float t[32];
            // 32 scores from position k0 on; a masked one is -inf
            auto take = [&](uint32_t addr, int k0) {
                uint32_t * v = reinterpret_cast<uint32_t *>(t);
                TMEM_LD32(addr, v);
                tmem_wait_ld();
                if (k0 + 31 > lim_min) {
#pragma unroll
                    for (int i = 0; i < 32; i++) t[i] = k0 + i <= lim ? t[i] : -INFINITY;
                }
            };
            float m = -INFINITY, base = 0.f;                                   // the row's reference (base: 0 while it has none), in units of log2
            double l = 0.0;
            float factor = 1.f;                                                // of the weights: 1 / sum for a row that has been looked at, 1 for others
            // weights of this thread's scores by the row's reference, their sum and the largest raw score
            auto weigh = [&](uint32_t addr, int k0, uint32_t * p, float & sum, float & top) {
                float e[4] = {0.f, 0.f, 0.f, 0.f}, tm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int h = 0; h < AT_COLS; h += 32) {
                    if (k0 + h > lim_max) {           // nothing of these 32 positions is visible to any row
#pragma unroll
                        for (int i = 0; i < 16; i++) p[h / 2 + i] = 0u;
                        continue;
                    }
                    take(addr + (uint32_t) h, k0 + h);
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const float a = ex2(fmaf(t[2 * i], c, -base)), b = ex2(fmaf(t[2 * i + 1], c, -base));
                        e[i & 1] += a;
                        e[2 + (i & 1)] += b;
                        tm[i & 3] = fmaxf(tm[i & 3], fmaxf(t[2 * i], t[2 * i + 1]));
                        p[h / 2 + i] = look > 0 ? pack_f16(a * factor, b * factor) : pack_f16(a, b);
                    }
                }
                sum = (e[0] + e[1]) + (e[2] + e[3]);
                top = fmaxf(fmaxf(tm[0], tm[1]), fmaxf(tm[2], tm[3]));
            };
            // the row's largest score of tile j, over both threads that hold the row, times scale * log2(e)
            auto row_top = [&](int j, float & top) {
                ctl->row_m[j & 1][part][row] = top;
                rows_barrier(quad);
                top = fmaxf(top, ctl->row_m[j & 1][part ^ 1][row]);
                top = top == -INFINITY ? top : top * c;
                return top;
            };
            if (look > 0) {
                for (int j = 0; j < look; j++) {
                    mbar_wait(&ctl->s_full, (tiles + looks + (uint32_t) j) & 1, cta_abort, P.abort_flag);
                    __syncwarp();
                    fence_after();
#pragma unroll
                    for (int h = 0; h < AT_COLS; h += 32) {
                        if (j * 128 + part * AT_COLS + h > lim_max) break;
                        take(mine + S0 + (uint32_t) h, j * 128 + part * AT_COLS + h);
                        float tm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, e[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int i = 0; i < 32; i++) tm[i & 3] = fmaxf(tm[i & 3], t[i]);
                        const float top = fmaxf(fmaxf(tm[0], tm[1]), fmaxf(tm[2], tm[3])), mn = fmaxf(m, top == -INFINITY ? top : top * c), at = mn == -INFINITY ? 0.f : mn;
#pragma unroll
                        for (int i = 0; i < 32; i++) e[i & 3] += ex2(fmaf(t[i], c, -at));   // a score that is no number reaches the sum
                        l = (m == -INFINITY ? l : l * (double) ex2(m - mn)) + (double) ((e[0] + e[1]) + (e[2] + e[3]));
                        m = mn;
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctl->s_free);
                }
                ctl->row_m[1][part][row] = m;
                ctl->row_l[part][row] = l;
                rows_barrier(quad);
                const float m2 = ctl->row_m[1][part ^ 1][row];
                const float top = fmaxf(m, m2);
                if (top != -INFINITY) l = (m == -INFINITY ? l : l * (double) ex2(m - top)) + (m2 == -INFINITY ? ctl->row_l[part ^ 1][row] : ctl->row_l[part ^ 1][row] * (double) ex2(m2 - top));
                else l += ctl->row_l[part ^ 1][row];
                const bool ends = lim < AT_EXACT;
                m = ends ? top : -INFINITY;
                base = m == -INFINITY ? 0.f : m;
                factor = !ends ? 1.f : lim >= 0 ? (float) (1.0 / l) : 0.f;
                l = 0.0;
            }
            for (int j = 0; j < n; j++) {   // to the end also once a wait has given up (all return at once then): the warps of a row meet in every tile
                mbar_wait(&ctl->s_full, (tiles + looks + (uint32_t) (look + j)) & 1, cta_abort, P.abort_flag);   // every P V in front has ended with it
                __syncwarp();
                fence_after();
                uint32_t p[AT_COLS / 2];
                float top = -INFINITY, sum = 0.f;
                bool again = j == 0;
                if (!again) {   // weights by the reference at hand, and the tile's largest score beside them
                    weigh(mine + S0, j * 128 + part * AT_COLS, p, sum, top);
                    again = __any_sync(0xffffffffu, row_top(j, top) > m + 8.f);
                } else {
#pragma unroll
                    for (int h = 0; h < AT_COLS; h += 32) {
                        if (part * AT_COLS + h > lim_max) break;
                        take(mine + S0 + (uint32_t) h, part * AT_COLS + h);
#pragma unroll
                        for (int i = 0; i < 32; i++) top = fmaxf(top, t[i]);
                    }
                    row_top(j, top);
                }
                if (again) {    // some row's score is beyond its reference by more than 2^8: the row takes it as its reference
                    const bool up = top > m + 8.f;
                    const float f = !up ? 1.f : m == -INFINITY ? 0.f : ex2(m - top);
                    if (up) { m = base = top; l *= (double) f; }
                    if (j > 0) {
#pragma unroll
                        for (int h = 0; h < AT_COLS; h += 32) {
                            uint32_t * v = reinterpret_cast<uint32_t *>(t);
                            TMEM_LD32(mine + O0 + (uint32_t) h, v);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; i++) t[i] *= f;
                            TMEM_ST16(mine + O0 + (uint32_t) h, v);
                            TMEM_ST16(mine + O0 + (uint32_t) (h + 16), v + 16);
                        }
                    }
                    weigh(mine + S0, j * 128 + part * AT_COLS, p, sum, top);
                }
                l += (double) sum;
                TMEM_ST16(mine + S0, p);              // over this thread's own scores
                TMEM_ST16(mine + S0 + 16u, p + 16);
                tmem_wait_st();
                if (j * 128 + 127 > lim_min) {
                    // the tile holds positions that some row does not see.  A weight of zero does not silence a value that is no number: positions no row
                    // sees are cleared (the cache may hold anything there), non-finite values that only later rows see are taken out and remembered
                    const uint32_t uv = loads + (uint32_t) (look + 2 * j + 1), s = uv % AT_STAGES;
                    mbar_wait(&ctl->full[s], (uv / AT_STAGES) & 1, cta_abort, P.abort_flag);
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
            ctl->row_l[part][row] = l;
            softmax_barrier();       // every warp has looked through its values
            l = 0.0;
#pragma unroll
            for (int i = 0; i < AT_PARTS; i++) l += ctl->row_l[i][row];
            const float inv = lim < AT_EXACT ? 1.f : (float) (1.0 / l);
            if (n > 0) {
                mbar_wait(&ctl->o_full, o_phase, cta_abort, P.abort_flag);
                __syncwarp();
                fence_after();
            } else {
                mbar_wait(&ctl->full[loads % AT_STAGES], (loads / AT_STAGES) & 1, cta_abort, P.abort_flag);   // key tile 0 is on its way into the ring all the same
            }
            // the result goes through the ring's memory (every tile has been used; row r's 16-byte pieces rotated by r) so that a warp stores whole rows
            float * os = reinterpret_cast<float *>(ring);
#pragma unroll
            for (int h = 0; h < AT_COLS; h += 32) {
                if (n > 0) {
                    uint32_t * v = reinterpret_cast<uint32_t *>(t);
                    TMEM_LD32(mine + O0 + (uint32_t) h, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i++) t[i] *= inv;
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
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");           // the next item's copies overwrite what was read and written here
        fence_before();
        __syncthreads();
        tiles += (uint32_t) n;
        looks += (uint32_t) look;
        loads += n > 0 ? (uint32_t) (look + 2 * n) : 1u;
        o_phase ^= n > 0 ? 1u : 0u;
    }
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
    constexpr size_t smem = 1024 + (size_t) (AT_STAGES + 1) * AT_STAGE + sizeof(AtCtl), alone = 116 * 1024;   // alone: more than half of an SM's
    static_assert(smem <= alone && 2 * alone > 232448, "shared memory of an SM");
    static FuncAttrCache cache;
    const cudaError_t e = ensure_dyn_smem(cache, (const void *) k_attn_prefill_tc, alone, true);
    if (e != cudaSuccess) return (int) e;
    const int gqa = n_head / n_head_kv;
    const float c = scale == 0.f ? FLT_MIN : fabsf(scale) * 1.4426950408889634f;   // a masked score stays -inf
    const int64_t items = (int64_t) ((n_tok + 128 / gqa - 1) / (128 / gqa)) * n_head_kv;
    if (items > INT32_MAX) return (int) cudaErrorInvalidValue;
    const AtParams P{q, out, pos_dev, n_head, n_head_kv, gqa, 128 / gqa, n_tok, (int) items, c, scale < 0.f ? -1.f : 1.f, abort_flag()};
    const int64_t ld = (int64_t) n_head_kv * 128;
    CUtensorMap mk, mv;
    int rc = make_map(mk, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, kcache, ld, n_kv_max, 1, ld, 0, 128);
    if (!rc) rc = make_map(mv, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, vcache, ld, n_kv_max, 1, ld, 0, 128);
    if (rc) return rc;
    const int64_t slots = 2 * (int64_t) sm_count();
    const bool spread = items <= sm_count();   // an SM for every item
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned) (items < slots ? items : slots));
    cfg.blockDim = dim3(AT_THREADS);
    cfg.dynamicSmemBytes = spread ? alone : smem;
    cfg.stream = st;
    // Barriers and tensor memory are set up while the kernel in front ends (the kernel waits before it reads anything), unless that could put two items on one SM while
    // others are idle, because the kernel in front is still there.  Where every item can have an SM of its own, shared memory for one CTA to an SM keeps them apart.
    // us in calls one after the other, 150 tokens / 250 / 512, waiting for the end of the kernel in front / this: 64 heads over 8 14.3 / 11.6, 14.4 / 11.8, - ; 32 over 8 12.0 / 11.0,
    // 12.8 / 11.4, 14.4 / 13.6 (two walks over the keys 12.3, 12.3, 17.8)
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = spread || items >= slots ? 1 : 0;
    return (int) cudaLaunchKernelEx(&cfg, k_attn_prefill_tc, mk, mv, P);
}

}  // namespace pb
