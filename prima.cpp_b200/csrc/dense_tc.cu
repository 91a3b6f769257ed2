// prima.cpp_b200/csrc/dense_tc.cu — bf16 dense product for decode batches and prompts on the 5th-generation tensor cores:
//   C[t][n] = alpha * sum_k A[t][k] W[n][k] (+ bias[n]) (+ resid[t][n]),   A [T][K], W [N][K] row-major bf16, C f32.
// Weight rows are the M side of tcgen05.mma (lane of the accumulator = weight row, so a warp of the epilogue stores 32 consecutive floats of
// one token's row), tokens the N side.  Both operands travel from their row-major layout into the swizzle-128B K-major shared-memory image by
// tiled TMA loads (one elected thread; rows and k beyond the matrix read zeros), one elected thread issues the MMAs, tcgen05.commit hands
// stages back.  Two kernels:
//   k_dense_pair   products that fill the machine: a CTA pair shares 256 weight rows x 256 tokens (cta_group::2), each CTA staging half of both
//                  operands, persistent over the tiles with two accumulators, so that a tile is read out while the next one is multiplied
//   k_dense_split  the others: 128 weight rows x BN tokens per CTA; a cluster of up to 8 CTAs cuts K into equal consecutive parts and adds the
//                  partial sums in the parts' order through distributed shared memory
// What bounds them: all SMs together take about 12.5 TB/s from L2, and a 64-k step of a tile loads (rows + tokens) * 128 bytes: 128 x 256 tiles
// are held to 0.65 of the tensor rate by that, the pair's 256 x 256 to 0.87; small batches are bound by the weights' way from HBM.  Measured
// (2048 x 28672 x 4096): 870 us with cp.async producers and 128 x 256 tiles before, 345 us with the pair, 389 in calls one by one under the power limit.  No atomics: the sum of an
// element has one order, fixed by (T, N, K).  Every wait is bounded (common.cuh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "launch.h"
#include "layers.h"
#include "mixers.cuh"
#include "tc.cuh"

namespace pb {
namespace {

constexpr int TC_BM = 128, TC_BK = 64, TC_MAX_STAGES = 10;
constexpr int TC_A_BYTES = TC_BM * 128;                       // one stage of weights: 128 rows x 64 bf16
constexpr int PAIR_BN = 256, PAIR_STAGES = 6, PAIR_THREADS = 320, PAIR_STAGE = TC_A_BYTES + PAIR_BN / 2 * 128;
constexpr int SPLIT_THREADS = 256, MAX_SPLIT = 8;

struct TcCtl {
    uint64_t full[TC_MAX_STAGES], empty[TC_MAX_STAGES], acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort;
};

struct TcParams {
    float * C; int64_t ldc;
    const float * bias; const float * resid; int64_t ldr;
    float alpha;
    int T, N, K;
    int * abort_flag;
    // grouped: rows [grp_start[g], + grp_count[g]) of A times the g-th matrix of W into the same rows of C.  The counts live on the device:
    // blockIdx.y numbers the token tiles of all groups in a row (group 0's tiles, then group 1's, ...), the grid has room for the most tiles
    // there can be (rows / BN + groups) and a CTA past the last tile leaves at once.
    const int32_t * grp_start; const int32_t * grp_count; int groups;
    int plane_rows;        // planes: weight rows [p * plane_rows, + plane_rows) meet the p-th operand (a multiple of the row tile)
    int splits;            // CTAs of a cluster that share a tile's K
    int row_tiles, tok_tiles;
    DenseAct act;
};

// epilogue of NT tokens t, t + 1, ... of the warp's 32 consecutive weight rows (lane: row n); v: the sums.  FULL: all NT tokens exist (the
// test per token is a fifth of the instructions, and instructions are what bounds this part: 46 a warp and stored row before the
// paths were split, 11 us of a 256-token tile).  Residuals are fetched together before the first store: C may be the same memory, and
// every load behind a store would wait for it.
struct Finish {
    float bias, xp, xn;
    int y0;   // grouped: row of act.y of the group's first token
    __device__ __forceinline__ Finish(const TcParams & P, int n, int first = 0) {
        y0 = first;
        bias = (P.bias && n < P.N) ? P.bias[n] : 0.f;
        xp = P.act.xielu ? softplus_f(P.act.xielu[0]) : 0.f;
        xn = P.act.xielu ? 0.5f + softplus_f(P.act.xielu[1]) : 0.f;
    }
    template <int NT, bool FULL>
    __device__ __forceinline__ void store(const TcParams & P, float * Cm, int n, int t, int Tn, const float (&v)[NT]) const {
        if (P.act.silu_glu) {   // neighbouring lanes hold a gate and its value: of two tokens the even lane finishes the first, the odd one the second
            const int odd = threadIdx.x & 1;
            __nv_bfloat16 * y = (__nv_bfloat16 *) P.act.y + (int64_t) (t + odd) * P.act.ldy + n / 2;
            const int64_t step = 2 * P.act.ldy;
#pragma unroll
            for (int i = 0; i < NT; i += 2, y += step) {
                const float v0 = P.alpha * v[i], v1 = i + 1 < NT ? P.alpha * v[i + 1 < NT ? i + 1 : 0] : 0.f;
                const float mine = odd ? v1 : v0, other = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
                const float g = odd ? other : mine, u = odd ? mine : other;
                // the fast exponential and quotient are far more accurate than the operand type the result is rounded to
                if (n < P.N && i + odd < NT && (FULL || t + i + odd < Tn)) *y = __float2bfloat16_rn(__fdividef(g, 1.f + __expf(-g)) * u);
            }
            return;
        }
        if (n >= P.N) return;
        if (P.act.relu2) {
            __nv_bfloat16 * y = (__nv_bfloat16 *) P.act.y + (int64_t) (y0 + t) * P.act.ldy + n;
#pragma unroll
            for (int i = 0; i < NT; i++, y += P.act.ldy)
                if (FULL || t + i < Tn) {
                    const float r = fmaxf(fmaf(P.alpha, v[i], bias), 0.f);
                    *y = __float2bfloat16_rn(r * r);
                }
            return;
        }
        if (P.act.xielu) {
            __nv_bfloat16 * y = (__nv_bfloat16 *) P.act.y + (int64_t) t * P.act.ldy + n;
#pragma unroll
            for (int i = 0; i < NT; i++, y += P.act.ldy)
                if (FULL || t + i < Tn) *y = __float2bfloat16_rn(xielu_f(fmaf(P.alpha, v[i], bias), xp, xn));
            return;
        }
        float * c = Cm + (int64_t) t * P.ldc + n;
        if (P.resid) {
            const float * rp = P.resid + (int64_t) t * P.ldr + n;
            float r[NT];
#pragma unroll
            for (int i = 0; i < NT; i++, rp += P.ldr) r[i] = FULL || t + i < Tn ? *rp : 0.f;
#pragma unroll
            for (int i = 0; i < NT; i++, c += P.ldc)
                if (FULL || t + i < Tn) *c = fmaf(P.alpha, v[i], bias) + r[i];
        } else {
#pragma unroll
            for (int i = 0; i < NT; i++, c += P.ldc)
                if (FULL || t + i < Tn) *c = fmaf(P.alpha, v[i], bias);
        }
    }
    // NT columns of the accumulator from column address `taddr` on
    template <int NT>
    __device__ __forceinline__ void columns(const TcParams & P, float * Cm, int n, int t, int Tn, uint32_t taddr) const {
        uint32_t v[NT];
        tmem_ld(taddr, v);
        float f[NT];
#pragma unroll
        for (int i = 0; i < NT; i++) f[i] = __uint_as_float(v[i]);
        if (t + NT <= Tn) store<NT, true>(P, Cm, n, t, Tn, f);
        else store<NT, false>(P, Cm, n, t, Tn, f);
    }
};

// ---------------------------------------------------------------------------------------------------------------
// 128 weight rows x BN tokens, K cut over the cluster.  Warp 0: TMA producer, warp 1: MMA issuer and owner of the TMEM columns; all 8 warps read
// the accumulator out (TMEM quadrant = warp % 4, token halves).
template <int BN, int STAGES>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
    k_dense_split(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ TcParams P) {
    constexpr int B_BYTES = BN * 128, STAGE = TC_A_BYTES + B_BYTES, COLS = BN < 32 ? 32 : BN;
    float * Cm = P.C;
    int Tn = P.T, tile_y = blockIdx.y, grp = 0, a_row0 = 0;
    if (P.grp_count) {
        pdl_wait();                    // the counts come from the kernels in front
        for (; grp < P.groups; grp++) {
            const int nt = (P.grp_count[grp] + BN - 1) / BN;
            if (tile_y < nt) break;
            tile_y -= nt;
        }
        if (grp >= P.groups) return;   // the whole cluster, before any barrier or TMEM allocation
        Tn = P.grp_count[grp];
        a_row0 = P.grp_start[grp];
        Cm += (int64_t) a_row0 * P.ldc;
    }
    extern __shared__ uint8_t smem_raw[];
    uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    TcCtl * ctl = reinterpret_cast<TcCtl *>(smem + STAGES * STAGE);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int S = P.splits, part = blockIdx.x % S;
    const int n0 = (blockIdx.x / S) * TC_BM, t0 = tile_y * BN;
    const int plane = P.plane_rows > 0 ? n0 / P.plane_rows : 0;
    const int nk = (P.K + TC_BK - 1) / TC_BK, u0 = nk * part / S, nu = nk * (part + 1) / S - u0;

    if (threadIdx.x == 0) {
        prefetch_map(&map_w);
        prefetch_map(&map_a);
        for (int i = 0; i < STAGES; i++) { mbar_init(&ctl->full[i], 1); mbar_init(&ctl->empty[i], 1); }
        mbar_init(&ctl->acc_full[0], 1);
        ctl->abort = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        pdl_trigger();   // behind the allocation: a later kernel's CTA on this SM must not take the columns first and wait for this one
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *(volatile uint32_t *) &ctl->tmem_base;
    volatile int * cta_abort = &ctl->abort;

    if (warp == 0) {
        // the weights of the first stages are on their way before the kernel in front has ended; its result is A
        const int ahead = min(nu, STAGES);
        auto load_w = [&](int u) {
            const int s = u % STAGES;
            mbar_arrive_expect_tx(&ctl->full[s], STAGE);
            tma_load<1>(smem_u32(smem + s * STAGE), &map_w, (u0 + u) * TC_BK, n0, grp, smem_u32(&ctl->full[s]));
        };
        auto load_a = [&](int u) {
            const int s = u % STAGES;
            tma_load<1>(smem_u32(smem + s * STAGE + TC_A_BYTES), &map_a, (u0 + u) * TC_BK, a_row0 + t0, plane, smem_u32(&ctl->full[s]));
        };
        if (elect_one())
            for (int u = 0; u < ahead; u++) load_w(u);
        __syncwarp();
        pdl_wait();
        if (elect_one())
            for (int u = 0; u < ahead; u++) load_a(u);
        __syncwarp();
        for (int u = ahead; u < nu; u++) {
            mbar_wait(&ctl->empty[u % STAGES], (uint32_t) ((u / STAGES - 1) & 1), cta_abort, P.abort_flag);
            __syncwarp();
            if (elect_one()) { load_w(u); load_a(u); }
            __syncwarp();
            if (*cta_abort) break;
        }
        __syncwarp();
    } else if (warp == 1) {
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (BN >> 3) << 17) | ((uint32_t) (TC_BM >> 4) << 24);
        for (int u = 0; u < nu; u++) {
            const int s = u % STAGES;
            mbar_wait(&ctl->full[s], (uint32_t) ((u / STAGES) & 1), cta_abort, P.abort_flag);
            __syncwarp();
            fence_after();
            const uint64_t da = desc_sw128(smem_u32(smem + s * STAGE)), db = desc_sw128(smem_u32(smem + s * STAGE + TC_A_BYTES));
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < TC_BK / 16; k++) mma_f16<1>(tmem, da + 2 * k, db + 2 * k, idesc, (uint32_t) ((u | k) != 0));
                mma_commit(&ctl->empty[s]);        // arrives once the MMAs above have read the stage
                if (u == nu - 1) mma_commit(&ctl->acc_full[0]);
            }
            __syncwarp();
        }
    }
    pdl_wait();                        // residual rows are read and results written behind it
    mbar_wait(&ctl->acc_full[0], 0u, cta_abort, P.abort_flag);
    __syncwarp();
    fence_after();
    {
        const int quad = warp & 3, half = warp >> 2, r = quad * 32 + lane, n = n0 + r;
        const Finish finish(P, n, a_row0);
        const uint32_t tq = tmem + ((uint32_t) (quad * 32) << 16);
        constexpr int HC = BN >= 32 ? BN / 2 : BN;   // columns per warp: halves of the tile, or all of a 16-token tile for the first four warps
        const int c_lo = half * HC, c_hi = c_lo + HC;
        if (S == 1) {
            for (int c0 = c_lo; c0 < c_hi && c0 < BN && t0 + c0 < Tn; c0 += 16) finish.template columns<16>(P, Cm, n, t0 + c0, Tn, tq + (uint32_t) c0);
        } else {
            // partial sums [token][row] in the stages' memory (every load and MMA of this CTA is done); token t is added up by CTA t % S
            float * red = reinterpret_cast<float *>(smem);
            for (int c0 = c_lo; c0 < c_hi && c0 < BN && t0 + c0 < Tn; c0 += 16) {
                uint32_t v[16];
                tmem_ld(tq + (uint32_t) c0, v);
#pragma unroll
                for (int i = 0; i < 16; i++) red[(c0 + i) * TC_BM + r] = __uint_as_float(v[i]);
            }
            __syncwarp();
            cluster_barrier();
            const int tn = min(BN, Tn - t0);
            for (int t = part + S * half; t < tn; t += 2 * S) {
                const uint32_t at = smem_u32(red + t * TC_BM + r);
                float f[MAX_SPLIT], v[1] = {0.f};
#pragma unroll
                for (int c = 0; c < MAX_SPLIT; c++) {
                    f[c] = 0.f;
                    if (c < S) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f[c]) : "r"(cluster_addr(at, (uint32_t) c)));
                }
#pragma unroll
                for (int c = 0; c < MAX_SPLIT; c++)
                    if (c < S) v[0] += f[c];
                finish.template store<1, true>(P, Cm, n, t0 + t, Tn, v);
            }
            __syncwarp();
            cluster_barrier();   // no CTA leaves while another one reads its partial sums
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------------------------
// CTA pair: 256 weight rows x 256 tokens a tile, tiles token-first so that the pairs at work share weight rows in L2.  The leader (rank 0) issues
// the MMAs of both; its full barriers count the bytes of both CTAs' loads.  Warp 0: TMA producer, warp 1: MMA issuer (leader), TMEM owner;
// warps 2 .. 9 read accumulators out.
__global__ void __launch_bounds__(PAIR_THREADS, 1) __cluster_dims__(2, 1, 1)
    k_dense_pair(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ TcParams P) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    TcCtl * ctl = reinterpret_cast<TcCtl *>(smem + PAIR_STAGES * PAIR_STAGE);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int tiles = P.row_tiles * P.tok_tiles;
    const int nk = (P.K + TC_BK - 1) / TC_BK;

    if (threadIdx.x == 0) {
        prefetch_map(&map_w);
        prefetch_map(&map_a);
        for (int i = 0; i < PAIR_STAGES; i++) { mbar_init(&ctl->full[i], 1); mbar_init(&ctl->empty[i], 1); }
        for (int i = 0; i < 2; i++) { mbar_init(&ctl->acc_full[i], 1); mbar_init(&ctl->acc_empty[i], 16); }
        ctl->abort = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        pdl_trigger();   // behind the allocation: a later kernel's CTA on this SM must not take the columns first and wait for this one
    }
    fence_before();
    __syncthreads();
    cluster_barrier();   // both CTAs' barriers exist before anything arrives on them from the other CTA
    fence_after();
    const uint32_t tmem = *(volatile uint32_t *) &ctl->tmem_base;
    volatile int * cta_abort = &ctl->abort;

    if (warp == 0) {
        int u = 0;
        const int ahead = pair < tiles ? min(nk, PAIR_STAGES) : 0;   // stages whose weights are on their way before the kernel in front has ended
        auto load_w = [&](int s, int k, int n0) {
            if (rank == 0) mbar_arrive_expect_tx(&ctl->full[s], 2 * PAIR_STAGE);
            tma_load<2>(smem_u32(smem + s * PAIR_STAGE), &map_w, k * TC_BK, n0 + rank * TC_BM, 0, cluster_addr(smem_u32(&ctl->full[s]), 0));
        };
        if (elect_one())
            for (int k = 0; k < ahead; k++) load_w(k, k, (pair / P.tok_tiles) * 2 * TC_BM);
        __syncwarp();
        pdl_wait();
        for (int i = pair; i < tiles && !*cta_abort; i += pairs) {
            const int n0 = (i / P.tok_tiles) * 2 * TC_BM, t0 = (i % P.tok_tiles) * PAIR_BN;
            const int plane = P.plane_rows > 0 ? n0 / P.plane_rows : 0;
            for (int k = 0; k < nk; k++, u++) {
                const int s = u % PAIR_STAGES;
                if (u >= PAIR_STAGES) mbar_wait(&ctl->empty[s], (uint32_t) ((u / PAIR_STAGES - 1) & 1), cta_abort, P.abort_flag);
                __syncwarp();
                if (elect_one()) {
                    if (u >= ahead) load_w(s, k, n0);
                    tma_load<2>(smem_u32(smem + s * PAIR_STAGE + TC_A_BYTES), &map_a, k * TC_BK, t0 + rank * (PAIR_BN / 2), plane, cluster_addr(smem_u32(&ctl->full[s]), 0));
                }
                __syncwarp();
                if (*cta_abort) break;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (PAIR_BN >> 3) << 17) | ((uint32_t) ((2 * TC_BM) >> 4) << 24);
            int u = 0, j = 0;
            for (int i = pair; i < tiles; i += pairs, j++) {
                const int buf = j & 1;
                if (j >= 2) mbar_wait(&ctl->acc_empty[buf], (uint32_t) ((j / 2 - 1) & 1), cta_abort, P.abort_flag);
                __syncwarp();
                if (*cta_abort) break;
                fence_after();
                for (int k = 0; k < nk; k++, u++) {
                    const int s = u % PAIR_STAGES;
                    mbar_wait(&ctl->full[s], (uint32_t) ((u / PAIR_STAGES) & 1), cta_abort, P.abort_flag);
                    __syncwarp();
                    fence_after();
                    const uint64_t da = desc_sw128(smem_u32(smem + s * PAIR_STAGE)), db = desc_sw128(smem_u32(smem + s * PAIR_STAGE + TC_A_BYTES));
                    if (elect_one()) {
#pragma unroll
                        for (int q = 0; q < TC_BK / 16; q++) mma_f16<2>(tmem + buf * PAIR_BN, da + 2 * q, db + 2 * q, idesc, (uint32_t) ((k | q) != 0));
                        mma_commit_pair(&ctl->empty[s]);
                        if (k == nk - 1) mma_commit_pair(&ctl->acc_full[buf]);
                    }
                    __syncwarp();
                }
            }
        }
        __syncwarp();
    } else {
        const int quad = warp & 3, half = (warp - 2) >> 2, r = quad * 32 + lane;
        int j = 0;
        pdl_wait();
        for (int i = pair; i < tiles; i += pairs, j++) {
            const int buf = j & 1;
            const int n = (i / P.tok_tiles) * 2 * TC_BM + rank * TC_BM + r, t0 = (i % P.tok_tiles) * PAIR_BN;
            const Finish finish(P, n);
            mbar_wait(&ctl->acc_full[buf], (uint32_t) ((j / 2) & 1), cta_abort, P.abort_flag);
            __syncwarp();
            fence_after();
            const uint32_t tq = tmem + ((uint32_t) (quad * 32) << 16) + (uint32_t) (buf * PAIR_BN);
            for (int c0 = half * (PAIR_BN / 2); c0 < (half + 1) * (PAIR_BN / 2) && t0 + c0 < P.T; c0 += 16)
                finish.template columns<16>(P, P.C, n, t0 + c0, P.T, tq + (uint32_t) c0);
            fence_before();
            __syncwarp();
            if (lane == 0)   // the leader may overwrite this accumulator
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr(smem_u32(&ctl->acc_empty[buf]), 0)) : "memory");
        }
    }
    fence_before();
    __syncthreads();
    cluster_barrier();   // the pair leaves together: MMAs, commits and loads of one CTA reach into the other's shared memory
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------------------------
struct TcOperands {
    const __nv_bfloat16 * A; int64_t lda, a_rows, a_planes, a_plane;
    const __nv_bfloat16 * W; int64_t ldw, w_rows, w_planes, w_plane;
};

template <int BN, int STAGES> constexpr size_t split_smem() { return 1024 + (size_t) STAGES * (TC_A_BYTES + BN * 128) + sizeof(TcCtl) + 64; }

template <int BN, int STAGES>
int launch_split_stages(const TcParams & P, const TcOperands & o, const dim3 & grid, cudaStream_t st) {
    static FuncAttrCache cache;
    const cudaError_t e = ensure_dyn_smem(cache, (const void *) k_dense_split<BN, STAGES>, split_smem<BN, STAGES>(), true);
    if (e != cudaSuccess) return (int) e;
    CUtensorMap mw, ma;
    int rc = make_map(mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, o.W, P.K, o.w_rows, o.w_planes, o.ldw, o.w_plane, TC_BM);
    if (!rc) rc = make_map(ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, o.A, P.K, o.a_rows, o.a_planes, o.lda, o.a_plane, BN);
    if (rc) return rc;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(SPLIT_THREADS);
    cfg.dynamicSmemBytes = split_smem<BN, STAGES>();
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned) P.splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_pdl ? 2 : 1;
    g_launches++;
    return (int) cudaLaunchKernelEx(&cfg, k_dense_split<BN, STAGES>, mw, ma, P);
}
// Stages: while every CTA has an SM to itself as many as fit; with more CTAs than SMs (at most 96 KB each) two of them share one, so that one's
// prologue and epilogue lie beside the other's loads.
int launch_split(int bn, TcParams P, const TcOperands & o, cudaStream_t st) {
    const dim3 grid((unsigned) ((P.N + TC_BM - 1) / TC_BM * P.splits), (unsigned) ((P.T + bn - 1) / bn + (P.grp_count ? P.groups : 0)));
    const bool shared = (int64_t) grid.x * grid.y > sm_count() || P.splits == MAX_SPLIT;
    switch (bn) {
    case 16: return shared ? launch_split_stages<16, 5>(P, o, grid, st) : launch_split_stages<16, 10>(P, o, grid, st);
    case 32: return shared ? launch_split_stages<32, 5>(P, o, grid, st) : launch_split_stages<32, 10>(P, o, grid, st);
    case 64: return shared ? launch_split_stages<64, 4>(P, o, grid, st) : launch_split_stages<64, 8>(P, o, grid, st);
    case 128: return shared ? launch_split_stages<128, 3>(P, o, grid, st) : launch_split_stages<128, 6>(P, o, grid, st);
    default: return launch_split_stages<256, 4>(P, o, grid, st);
    }
}
int launch_pair(TcParams P, const TcOperands & o, cudaStream_t st) {
    constexpr size_t smem = 1024 + (size_t) PAIR_STAGES * PAIR_STAGE + sizeof(TcCtl) + 64;
    static FuncAttrCache cache;
    const cudaError_t e = ensure_dyn_smem(cache, (const void *) k_dense_pair, smem, true);
    if (e != cudaSuccess) return (int) e;
    P.row_tiles = (P.N + 2 * TC_BM - 1) / (2 * TC_BM);
    P.tok_tiles = (P.T + PAIR_BN - 1) / PAIR_BN;
    CUtensorMap mw, ma;
    int rc = make_map(mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, o.W, P.K, o.w_rows, o.w_planes, o.ldw, o.w_plane, TC_BM);
    if (!rc) rc = make_map(ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, o.A, P.K, o.a_rows, o.a_planes, o.lda, o.a_plane, PAIR_BN / 2);
    if (rc) return rc;
    const int64_t tiles = (int64_t) P.row_tiles * P.tok_tiles;
    const int pairs = (int) (tiles < sm_count() / 2 ? tiles : sm_count() / 2);
    g_launches++;
    return launch_dep(k_dense_pair, dim3((unsigned) (2 * pairs)), dim3(PAIR_THREADS), smem, st, mw, ma, P);
}

// Which kernel, token tile and cut of K: the one with the least time by a model of what was measured on a B200 (148 SMs, 1.9 GHz, all tiles of
// T 8 .. 2048, N 256 .. 32000, K 512 .. 14336, launches back to back in a graph; within 15 % of every time):
//   an SM takes 0.2 us for a 64-k step of one tile up to 128 tokens wide (what issuing and waiting cost), 0.28 us for 256 (its MMAs);
//   all SMs together take 12.5 TB/s from L2 and 6.5 TB/s of weights from HBM;
//   a launch costs 3 us + 0.01 us per token of the tile (9 us with the pair's two accumulators), a cut of K 1.5 us + 0.015 us per token more.
// Examples, us: 8 x 2048 x 8192 uncut 37.9, cut in 4 13.7, in 8 10.6; 512 x 2048 x 8192 pair 47.4, 128 tokens 31.2, cut in 4 24.1;
// 1488 x 16384 x 2048 pair 81.8, 256 tokens 105, 128 tokens 119.  rows: tokens (grouped: expected ones of a group).
struct TcPlan { int pair, bn, splits; };
TcPlan plan_tc(int rows, int groups, int N, int K, int plane_rows) {
    const int64_t nk = (K + TC_BK - 1) / TC_BK, sms = sm_count();
    const double hbm = (double) N * K * 2 * groups / 6.5e6;
    TcPlan best{0, 64, 1};
    double best_us = 1e30;
    auto consider = [&](const TcPlan & p, int64_t steps_of_an_sm, double step_us, int64_t steps, int step_bytes, double fixed_us) {
        const double us = std::max({(double) steps_of_an_sm * step_us, (double) steps * step_bytes / 12.5e6, hbm}) + fixed_us;
        if (us <= best_us) { best_us = us; best = p; }   // of equals the finer cut: two CTAs to an SM hide each other's start and end
    };
    if (groups == 1 && rows > 128 && plane_rows % (2 * TC_BM) == 0) {
        const int64_t tiles = (int64_t) ((N + 2 * TC_BM - 1) / (2 * TC_BM)) * ((rows + PAIR_BN - 1) / PAIR_BN), waves = (tiles + sms / 2 - 1) / (sms / 2);
        consider({1, PAIR_BN, 1}, waves * nk, 0.28, tiles * nk, 2 * PAIR_STAGE, 9.0);
    }
    for (int bn = 16; bn <= 256; bn *= 2) {
        if (bn > 16 && rows <= bn / 2) break;
        const int64_t tiles = (int64_t) ((N + TC_BM - 1) / TC_BM) * ((rows + bn - 1) / bn) * groups;
        for (int s = 1; s <= MAX_SPLIT && s <= nk; s *= 2) {
            if (s > 1 && (bn > 128 || groups > 1 || tiles * s > 2 * sms)) break;
            const int64_t per_sm = (tiles * s + sms - 1) / sms;
            consider({0, bn, s}, per_sm * ((nk + s - 1) / s), bn > 128 ? 0.28 : 0.2, tiles * nk, (TC_BM + bn) * 128,
                     3.0 + 0.01 * bn + (s > 1 ? 1.5 + 0.015 * bn : 0.0) + (bn > 128 ? 2.5 * (double) (per_sm - 1) : 0.0));
        }
    }
    return best;
}

}  // namespace

bool dense_tc_ok(int T, int N, int K, int64_t lda, int64_t ldw, const void * A, const void * W) {
    static const bool off = getenv("PB200_NO_DENSE_TC") != nullptr;   // A/B: the CUDA-core tile kernel instead
    return !off && T > 0 && N > 0 && K >= 8 && K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && ((uintptr_t) A & 15) == 0 && ((uintptr_t) W & 15) == 0;
}

int launch_dense_tc(const __nv_bfloat16 * A, int64_t lda, const __nv_bfloat16 * W, int64_t ldw, float * C, int64_t ldc, int T, int N, int K, const float * bias,
                    const float * resid, int64_t ldr, float alpha, cudaStream_t st, int plane_rows, int64_t a_plane, DenseAct act) {
    TcParams P{C, ldc, bias, resid, ldr, alpha, T, N, K, abort_flag(), nullptr, nullptr, 1, plane_rows, 1, 0, 0, act};
    const TcOperands o{A, lda, T, plane_rows > 0 ? N / plane_rows : 1, a_plane, W, ldw, N, 1, 0};
    const TcPlan p = plan_tc(T, 1, N, K, plane_rows);
    if (p.pair) return launch_pair(P, o, st);
    P.splits = p.splits;
    return launch_split(p.bn, P, o, st);
}

int launch_dense_tc_grouped(const __nv_bfloat16 * A, int64_t lda, const __nv_bfloat16 * W, int64_t ldw, int64_t w_stride, float * C, int64_t ldc,
                            const int32_t * start, const int32_t * count, int groups, int max_rows, int N, int K, cudaStream_t st, DenseAct act) {
    if (groups <= 0 || max_rows <= 0) return 0;
    // T bounds the grid only (all groups together hold max_rows rows); the kernel reads each group's own count
    TcParams P{C, ldc, nullptr, nullptr, 0, 1.f, max_rows, N, K, abort_flag(), start, count, groups, 0, 1, 0, 0, act};
    const TcOperands o{A, lda, max_rows, 1, 0, W, ldw, N, groups, w_stride};
    const TcPlan p = plan_tc((max_rows + groups - 1) / groups, groups, N, K, 0);   // the tile follows the expected rows of a group
    P.splits = 1;
    return launch_split(p.bn, P, o, st);
}

}  // namespace pb
