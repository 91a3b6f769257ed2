// prima.cpp_b200/csrc/mmq.cu — batched (prefill) k-quant mat-mul on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// Replaces: ggml_cuda_op_mul_mat_q -> mul_mat_q<type,mmq_x,8,chk> (ggml-cuda/mmq.cu:3-98, mmq.cuh:2583-2650: int8 mma.sync
// tiles with __syncthreads ping-pong) and quantize_mmq_q8_1_cuda (quantize.cu:143-169).
// Numerics follow the CPU backend the oracle restates: every activation row is quantized to q8_K exactly as
// quantize_row_q8_K_ref does (ggml-quants.c:3785-3822) and the weights are expanded with the dequantize_row_q{4,5,6}_K
// formulas (ggml-quants.c:2040-2065, 2390-2420, 2690-2725) evaluated in fp16 (exact integer q, fp16 sub-block scale and
// offset, one fused multiply-add); both operands are fp16 on the tensor pipe with fp32 accumulation.  The result differs
// from the integer-dot CPU value by a few fp16 roundings per product (NMSE ~1e-6; tests/test_gpu_mmq.py states the bound).
//
//   dst[t][n] = sum_k W[n][k] * X[t][k]        W: N x K k-quant rows, X: T x K f32, dst: T x N f32 (ggml layout)
// Also the 32-element block types Q8_0 / Q5_1 (K % 64 == 0; activations quantized per 32 values like their CPU dot): Qwen2.5-72B's
// ffn_down, whose K = 29 568 rules the k-quants out (src/llama.cpp:19516-19551).
//
// Work decomposition.  A work UNIT = one 256-element K group of one output tile (128 weight rows x 1 or 2 token tiles of BN <= 256 columns: two
// accumulators = all 512 TMEM columns share every expanded weight stage when T is large enough).  Two forms, chosen by mmq_pick_cut:
//   shares   the units of a launch, ordered tile by tile, are cut into one contiguous range per CTA (at most one CTA per SM), so that few SMs are
//            idle in a last wave.  A CTA walks its range segment by segment (segment = its part of one tile); a segment that covers the
//            tile's whole K stores its result, a partial one adds it into the pre-zeroed dst with fp32 atomics; a tile has two such
//            segments at most
//   cut      few tiles: a cluster of up to 8 CTAs shares one tile, each takes a part of its K, and the parts' sums are added in order through
//            distributed shared memory
// Either way an element's sum has one order: equal calls give equal bits.
// Inside a CTA the pipeline never drains between segments (raw-block ring, A and B stages and their barriers run on CTA-wide counters):
//   warp 0      owns TMEM; one lane issues 4 x tcgen05.mma (M=128, N=BN, K=16, kind::f16) per step and accumulator, one commit per step
//   warp 1      activation producer: one cp.async.bulk per step and accumulator of the pre-tiled fp16 chunk (BN x 128 B, already in the
//               UMMA swizzle-128B image), 2-4 stages deep
//   warp 18     fetches the rows' raw quantized blocks, a K group of the tile as one TMA box, 3 groups deep (rows that do not lie at multiples of 16
//               bytes: the expansion warps fetch them in 16-byte cp.async pieces)
//   warps 2..17 (16 expansion warps, 4 threads per weight row) take a group's blocks into registers (Q4_K, Q5_K: header and quants at once) and expand 128 x 64 weights per step to fp16 straight into the swizzled A
//               stage (generic-proxy stores + fence.proxy.async), 2 stages (4 with CTA pairs); at the end of a segment or part all 16 read the
//               accumulators out of TMEM (tcgen05.ld 32x32b: quadrant = warp % 4, every fourth chunk of 16 columns) and store / add into dst
// What bounds it: with two accumulators the tensor pipe (a step takes 1424 clocks, its eight M = 128, N = 256 MMAs 1368); with one, the chain of waits, fence
// and commit of a step (1050 clocks at 64 tokens).  14336 x 4096 at 512 tokens, Q4_K, raw blocks and scales by every thread -> by boxes and groups: 173 -> 126
// instructions a warp and step, 69.5 -> 67 us; Q6_K 4096 x 14336 73.5 -> 71; a group with few tokens 2.7 -> 2.3 us.
// CG = 2 (opt-in): the CTA pair of a cluster shares one M = 256 MMA (cta_group::2), see launch_mmq.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "launch.h"
#include "tc.cuh"

namespace pb {

constexpr int MMQ_BM = 128;
constexpr int MMQ_BK = 64;
constexpr int MMQ_A_MAX = 4;      // expanded-weight stages: P.a_nst = 2 or 4 (a power of two) of 16 KB, chosen at launch from the shared-memory budget
constexpr int MMQ_B_NST = 4;      // activation stages (L2 loads: the deep ring)
constexpr int MMQ_DQ_WARPS = 16;  // expansion warps: 4 threads per weight row, 16 weights per thread and step (8 warps were the latency-bound bottleneck: 45 % tensor pipe)
constexpr int MMQ_DQ_WARP0 = 2;   // warps 0,1 = MMA issuer (owns TMEM), activation producer
constexpr int MMQ_RAW_WARP = MMQ_DQ_WARP0 + MMQ_DQ_WARPS;   // fetches the raw blocks by tiled TMA
constexpr int MMQ_THREADS = (MMQ_RAW_WARP + 1) * 32;
constexpr int MMQ_A_BYTES = MMQ_BM * 128;   // one A stage: 128 rows x 64 fp16
constexpr int MMQ_CTL_BYTES = 320;
constexpr int MMQ_MAX_PARTS = 8;  // CTAs of a cluster that share a tile's K

struct MmqParams {
    int * abort_flag;      // host-mapped, raised by the wait watchdog
    const uint8_t * W;
    const uint8_t * B;     // activations, fp16, tiled [T/BN][K/64][BN x 128 B swizzled]
    float * dst;           // [T][N]
    const float * bias;    // [N] or null
    const float * resid;   // [T][N] or null: residual added in the epilogue
    int64_t row_bytes, total_bytes;
    int nraw, b_nst, a_nst;   // ring depths chosen at launch from the shared-memory budget (a_nst: 2 or 4)
    int nacc, ttiles;      // accumulators (token tiles) per output tile, number of token tiles
    int ngrp, rtiles;      // 256-K groups per row (the last one may be short: 32-element block types), row tiles
    int parts;             // > 1: the CTAs of a cluster, one tile each cluster, share the tile's K groups; else
    int upc, total_units;  // work units per CTA (CTA c owns units [c * upc, min((c + 1) * upc, total_units)) ), units of the launch
    int tma;               // the raw blocks come by tiled TMA; 0: rows that do not lie at multiples of 16 bytes, fetched by the expansion warps
    int chain;             // > 0: instead, chains of that many tiles (the last one: what is left), each in equal shares for one CTA more than it has tiles
    int N, K, T, BN, bpb, slot;   // slot: bytes reserved per row in a raw stage (16-B aligned window around one block)
    uint32_t tmem_cols, idesc;
};

// Several matrices over one activation in a cut launch: row tiles [rt0, next rt0) belong to a matrix.  `slot` as in MmqParams; `second`: its blocks are of the
// kernel's second type.
constexpr int MMQ_MAX_MATS = 3;
struct MmqMat {
    const uint8_t * W;
    float * dst;
    const float * bias;
    int64_t row_bytes, total_bytes;
    int N, rt0, bpb, slot, second;
};
template <bool MULTI> struct MmqMats { CUtensorMap map[1]; };
template <> struct MmqMats<true> { CUtensorMap map[MMQ_MAX_MATS]; MmqMat mat[MMQ_MAX_MATS]; int n; };

struct MmqCtl {
    uint64_t raw_full[3], raw_empty[3];
    uint64_t a_ready[MMQ_A_MAX], b_full[MMQ_B_NST];
    uint64_t step_done[MMQ_B_NST];   // one tcgen05.commit per step: step u arrives on step_done[u % 4]; frees A stage u % 2 and B stage u % b_nst
    uint64_t acc_ready, acc_free;    // per segment: accumulators complete (tcgen05.commit) / read out by the 16 expansion warps (of both CTAs of a pair)
    uint64_t peer_ready[MMQ_B_NST];  // CTA pairs: step g's A and B stages of the peer CTA are filled (forwarded by the peer's otherwise idle warp 0)
    uint32_t tmem_base;
    volatile int abort;
};
static_assert(sizeof(MmqCtl) <= MMQ_CTL_BYTES, "ctl");


__device__ __forceinline__ bool mmq_try(uint64_t * bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait: a broken pipeline must end the launch (and report through pb200_mmq_aborted), never hang the device
__device__ __forceinline__ bool mmq_wait_(MmqCtl * ctl, uint64_t * bar, uint32_t parity, int * abort_flag) {
    if (mmq_try(bar, parity)) return true;          // the common case costs one try_wait
    const long long t0 = clock64();
    int spins = 0;
    while (!mmq_try(bar, parity)) {
        if ((++spins & 255) == 0) {
            if (ctl->abort) return false;
            if (clock64() - t0 > PB_WAIT_TIMEOUT_CYCLES) {
                ctl->abort = 1;                                          // inline on purpose: a call in this kernel costs 7-12 registers
                if (abort_flag) *(volatile int *) abort_flag = 1;        // host-mapped; visible at the latest when the launch ends
                return false;
            }
        }
    }
    return true;
}
#define mmq_wait(ctl, bar, parity) mmq_wait_(ctl, bar, parity, P.abort_flag)
__device__ __forceinline__ void bulk_g2s_plain(void * smem_dst, const void * gsrc, uint32_t bytes, uint64_t * bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)), "l"(gsrc),
                 "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    // K-major, SWIZZLE_128B: rows of 128 B, 8-row groups 1024 B apart (cute/arch/mma_sm100_desc.hpp SmemDescriptor)
    uint64_t d = (uint64_t) ((saddr >> 4) & 0x3FFF);
    d |= (uint64_t) 1 << 16;               // leading byte offset: unused for swizzled K-major, canonical value 1
    d |= (uint64_t) (1024 >> 4) << 32;     // stride byte offset
    d |= (uint64_t) 1 << 46;               // descriptor version (Blackwell)
    d |= (uint64_t) 2 << 61;               // SWIZZLE_128B
    return d;
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t * bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// cta_group::2: the CTA pair of a cluster executes one M = 256 MMA; A rows 0-127 / 128-255 and the two halves of B's N rows come from the two
// CTAs' shared memory at the same offsets, each CTA's TMEM receives its own 128 rows of D.  Issued by the leader CTA (rank 0) only.
__device__ __forceinline__ void umma_f16_cg2(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// completion of all prior MMAs of the pair -> the barrier at this offset in BOTH CTAs
__device__ __forceinline__ void umma_commit_cg2(uint64_t * bar) {
    const uint16_t mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(mask)
                 : "memory");
}
__device__ __forceinline__ uint32_t mmq_cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void mmq_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// what every thread of the cluster has loaded from the others' shared memory is in its registers: nothing is published
__device__ __forceinline__ void mmq_cluster_read() {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}
// a shared-memory address of this CTA in CTA `rank` of the cluster, and the float there
__device__ __forceinline__ uint32_t mmq_peer_addr(uint32_t saddr, uint32_t rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(saddr), "r"(rank));
    return ra;
}
__device__ __forceinline__ float mmq_peer_f32(uint32_t ra) {
    float f;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(ra) : "memory");
    return f;
}
// arrive on the barrier at the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t * bar, uint32_t rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(bar)), "r"(rank));
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(ra) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}
// 32-bit load from shared memory at an address that is only 2-byte aligned
__device__ __forceinline__ uint32_t lds32_u2(const uint8_t * p) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t * w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t) 3);
    if ((a & 2) == 0) return w[0];
    return __funnelshift_r(w[0], w[1], 16);
}

// ---- weight expansion: thread (row, h) produces K elements [64c + 32h, 64c + 32h + 32) of its row as 16 half2 ----
// The integer q of every weight is made an EXACT fp16 with the exponent trick (0x6400 | q == 1024 + q, minus 1024 + zero),
// then one half2 FMA applies the sub-block scale and offset (both rounded to fp16).  A 32-bit word holds 4 consecutive-k
// bytes; the two half2 come out as (k0,k2) and (k1,k3): the activation tiles use the same within-4 order (k_mmq_prep).
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t magic) {   // (a & mask) | magic in one LOP3
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(mask), "r"(magic));
    return d;
}
template <uint32_t MASK>
__device__ __forceinline__ void expand_word(uint32_t t, __half2 bias, __half2 scale, __half2 off, uint32_t & o02, uint32_t & o13) {
    const uint32_t p02 = and_or(t, MASK, 0x64006400u);
    const uint32_t p13 = and_or(t >> 8, MASK, 0x64006400u);
    o02 = h2_bits(__hfma2(__hadd2(bits_h2(p02), bias), scale, off));
    o13 = h2_bits(__hfma2(__hadd2(bits_h2(p13), bias), scale, off));
}
// thread (row, h, hh) produces K elements [64c + 32h + 16hh, 64c + 32h + 16hh + 16) of its row as 8 half2 (two 16-byte pieces of the A stage)
template <int TYPE>
__device__ __forceinline__ void expand(const uint8_t * blk, int c, int h, int hh, uint32_t (&out)[8]) {
    if (TYPE == T_Q8_0) {
        // 32-element blocks, 34 B each ([d f16][32 x i8]); blk = the group of 8 blocks covering 256 K, this thread's block is 2c + h.
        // Blocks are 2-byte aligned: qs (offset 2) is either word-aligned or straddles words -> one PRMT per word.
        const uint8_t * bb = blk + (2 * c + h) * BYTES_Q8_0;
        const uint32_t * wp = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(bb) & ~(uintptr_t) 3);
        const bool odd = (reinterpret_cast<uintptr_t>(bb) & 2) != 0;
        const uint32_t sel = odd ? 0x7654u : 0x5432u;
        const uint32_t w0 = wp[0];
        uint32_t w[5];
#pragma unroll
        for (int i = 0; i < 5; i++) w[i] = wp[4 * hh + i];
        const __half dh = __ushort_as_half((unsigned short) ((w0 >> (odd ? 16 : 0)) & 0xffff));
        const __half2 scale = __half2half2(dh), bias = __float2half2_rn(-1152.f), zero = __float2half2_rn(0.f);
#pragma unroll
        for (int i = 0; i < 4; i++)   // q + 128 as an unsigned byte, 0x6400 | u = 1024 + u, minus 1152 = q exactly
            expand_word<0x00FF00FFu>(__byte_perm(w[i], w[i + 1], sel) ^ 0x80808080u, bias, scale, zero, out[2 * i], out[2 * i + 1]);
    } else if (TYPE == T_Q5_1) {
        // 24 B blocks ([d f16][m f16][qh u32][16 x 2 nibbles]), 8-byte aligned; element j < 16 = low nibble of qs[j] | bit j of qh << 4,
        // element j + 16 = high nibble | bit j + 16: hh = 0 takes the low nibbles, hh = 1 the high ones
        const uint8_t * bb = blk + (2 * c + h) * BYTES_Q5_1;
        const uint2 hd = *reinterpret_cast<const uint2 *>(bb);
        const __half2 dm = bits_h2(hd.x);
        const __half2 scale = __half2half2(__low2half(dm)), off = __half2half2(__high2half(dm)), bias = __float2half2_rn(-1024.f);
        const uint32_t qh = hd.y >> (16 * hh);
        const uint2 qa = *reinterpret_cast<const uint2 *>(bb + 8), qb = *reinterpret_cast<const uint2 *>(bb + 16);
        const uint32_t w[4] = {qa.x, qa.y, qb.x, qb.y};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t hb = ((((qh >> (4 * i)) & 0xFu) * 0x00204081u) & 0x01010101u) << 4;
            expand_word<0x001F001Fu>(((w[i] >> (4 * hh)) & 0x0F0F0F0Fu) | hb, bias, scale, off, out[2 * i], out[2 * i + 1]);
        }
    } else {
        // Q6_K: blk is 2-byte aligned only (210-byte blocks): words are fetched as aligned pairs and funnel-shifted
        const float d = __half2float(*reinterpret_cast<const __half *>(blk + 208));
        const int n = c >> 1, p = c & 1;
        const uint8_t * ql = blk + 64 * n + 32 * h + 16 * hh;
        const uint8_t * qh = blk + 128 + 32 * n + 16 * hh;
        const int8_t * sc = reinterpret_cast<const int8_t *>(blk + 192 + 8 * n + 2 * h + 4 * p);
        const __half2 sca = __float2half2_rn(__fmul_rn(d, (float) sc[hh]));
        const __half2 bias = __float2half2_rn(-1056.f), zero = __float2half2_rn(0.f);
        const uint32_t shl = (uint32_t) (reinterpret_cast<uintptr_t>(blk) & 2) * 8;     // 0 or 16 (ql and qh share blk's alignment)
        const uint32_t * lw = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(ql) & ~(uintptr_t) 3);
        const uint32_t * hw = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(qh) & ~(uintptr_t) 3);
        uint32_t lprev = lw[0], hprev = hw[0];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t lnext = lw[i + 1], hnext = hw[i + 1];
            const uint32_t l = __funnelshift_r(lprev, lnext, shl), hq = __funnelshift_r(hprev, hnext, shl);
            lprev = lnext; hprev = hnext;
            const uint32_t t = ((l >> (4 * p)) & 0x0F0F0F0Fu) | (((hq >> (4 * p + 2 * h)) << 4) & 0x30303030u);
            expand_word<0x003F003Fu>(t, bias, sca, zero, out[2 * i], out[2 * i + 1]);
        }
    }
}

// Q4_K / Q5_K: what a thread takes of its row's block, all four steps of it: scales and offsets of the sub-blocks 2c + h (get_scale_min_k4, ggml-quants.c:1950-1958, for
// four bytes at a time; byte 2 (c & 1) of word c / 2 is step c's), the quants' words and for Q5_K the words of the fifth bits.  The header so is one load of a group and not five a step.
template <int TYPE>
struct KGroup {
    float d, dmin;
    uint32_t s[2], m[2], hb[4];
    uint4 q[4];
    __device__ __forceinline__ void load(const uint8_t * blk, int h, int hh) {
        const uint4 hd = *reinterpret_cast<const uint4 *>(blk);
#pragma unroll
        for (int c = 0; c < 4; c++) q[c] = *reinterpret_cast<const uint4 *>(blk + (TYPE == T_Q4_K ? 16 : 48) + 32 * c + 16 * hh);
        if (TYPE == T_Q5_K) {
            const uint4 b = *reinterpret_cast<const uint4 *>(blk + 16 + 16 * hh);
            hb[0] = b.x >> h; hb[1] = b.y >> h; hb[2] = b.z >> h; hb[3] = b.w >> h;
        }
        const __half2 dm = bits_h2(hd.x);
        d = __low2float(dm);
        dmin = __high2float(dm);
        s[0] = (hd.y & 0x3f3f3f3fu) >> (8 * h);
        m[0] = (hd.z & 0x3f3f3f3fu) >> (8 * h);
        s[1] = ((hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u)) >> (8 * h);
        m[1] = (((hd.w >> 4) & 0x0f0f0f0fu) | ((hd.z >> 2) & 0x30303030u)) >> (8 * h);
    }
    // What has been loaded is in registers (common.cuh): without this, blocks came out as a mixture of this group and the one that follows in the slot, where the activations
    // were late and all 16 warps went on together.
    __device__ __forceinline__ void loaded() const {
        uint32_t w = q[0].x ^ q[1].x ^ q[2].x ^ q[3].x ^ s[0];
        if (TYPE == T_Q5_K) w ^= hb[0];
        loads_done(w);
    }
    static __device__ __forceinline__ float byte_f(uint32_t w, int c) {   // exact: 2^23 + byte less 2^23
        return __fadd_rn(__uint_as_float(and_or((c & 1) ? w >> 16 : w, 0xffu, 0x4b000000u)), -8388608.f);
    }
    __device__ __forceinline__ void expand(int c, int h, uint32_t (&out)[8]) const {
        const __half2 so = __floats2half2_rn(__fmul_rn(d, byte_f(s[c >> 1], c)), -__fmul_rn(dmin, byte_f(m[c >> 1], c)));
        const __half2 scale = __low2half2(so), off = __high2half2(so);
        const uint32_t w[4] = {q[c].x, q[c].y, q[c].z, q[c].w};
        // a nibble in the low place makes 1024 + q, one in the high place 64 + q (0x5400 = 64, steps of 1 / 16)
        const uint32_t mask = h ? 0x00F000F0u : 0x000F000Fu, magic = h ? 0x54005400u : 0x64006400u;
        const __half2 bias = TYPE == T_Q5_K ? __float2half2_rn(-1024.f) : bits_h2(h ? 0xD400D400u : 0xE400E400u);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (TYPE == T_Q4_K) {
                const uint32_t p02 = (w[i] & mask) | magic, p13 = ((w[i] >> 8) & mask) | magic;
                out[2 * i] = h2_bits(__hfma2(__hadd2(bits_h2(p02), bias), scale, off));
                out[2 * i + 1] = h2_bits(__hfma2(__hadd2(bits_h2(p13), bias), scale, off));
            } else {
                const uint32_t fifth = c < 2 ? hb[i] << (4 - 2 * c) : hb[i] >> (2 * c - 4);
                expand_word<0x001F001Fu>(((w[i] >> (4 * h)) & 0x0F0F0F0Fu) | (fifth & 0x10101010u), bias, scale, off, out[2 * i], out[2 * i + 1]);
            }
        }
    }
};

__device__ __forceinline__ void tma_raw(uint32_t dst, const CUtensorMap * m, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(m), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(void * smem_dst, const void * gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}

// TYPE2 > 0 (cut launches): several matrices, whose blocks are of TYPE or TYPE2
template <int TYPE, int CG, bool CUT, int TYPE2 = 0>
__global__ void __launch_bounds__(MMQ_THREADS, 1) k_mmq_tc(const __grid_constant__ MmqParams P, const __grid_constant__ MmqMats<(TYPE2 > 0)> mm) {
    constexpr bool MULTI = TYPE2 > 0, MIXED = MULTI && TYPE2 != TYPE;
    static_assert(!MULTI || (CUT && CG == 1), "a CTA of a launch of several matrices walks one tile");
    extern __shared__ uint8_t smem_raw[];
    // the swizzle-128B atoms (A and B stages) need 1024-byte alignment in the shared window
    uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int BN = P.BN;
    const int b1 = BN * 128;                                     // one token tile's chunk in the activation image
    const int b1c = b1 / CG;                                     // this CTA's part of it: BN / CG token rows (a pair splits B's N rows)
    const int b_bytes = P.nacc * b1c;                            // one B stage
    const uint32_t rank = CG == 2 ? mmq_cluster_rank() : 0u;     // CTA pairs: rank 0 leads (issues the MMAs), rank 1 expands the tile's other 128 rows
    uint8_t * a_st = smem;                                       // [A_NST][16 KB]
    uint8_t * b_st = a_st + P.a_nst * MMQ_A_BYTES;               // [b_nst][nacc][BN/CG*128]
    const int amask = P.a_nst - 1, ashift = P.a_nst == 4 ? 2 : 1;
    uint8_t * raw = b_st + P.b_nst * b_bytes;                    // [nraw][128 * slot]
    MmqCtl * ctl = reinterpret_cast<MmqCtl *>(raw + P.nraw * MMQ_BM * P.slot);

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int nstep_all = P.K / MMQ_BK;                          // 64-element steps of a whole row; group sb holds steps [4 sb, min(4 sb + 4, nstep_all))
    // this CTA's (pair's) units; CUT: the part-th of a tile's equal consecutive parts, one segment
    const int part = CUT ? (int) blockIdx.x % P.parts : 0, cut0 = CUT ? (int) blockIdx.x / P.parts * P.ngrp : 0;
    int w0 = CUT ? cut0 + P.ngrp * part / P.parts : (int) (blockIdx.x / CG) * P.upc;
    int w1 = CUT ? cut0 + P.ngrp * (part + 1) / P.parts : min(w0 + P.upc, P.total_units);
    if (!CUT && P.chain > 0) {
        const int b = (int) blockIdx.x / CG, c = b / (P.chain + 1), j = b - c * (P.chain + 1), u0 = c * P.chain * P.ngrp;
        const int units = min(P.chain * P.ngrp, P.total_units - u0), shares = units / P.ngrp + 1;
        w0 = u0 + (int) ((int64_t) units * min(j, shares) / shares);
        w1 = u0 + (int) ((int64_t) units * min(j + 1, shares) / shares);
    }

    // the matrix: the only one, or that of this CTA's tile
    MmqMat M{P.W, P.dst, P.bias, P.row_bytes, P.total_bytes, P.N, 0, P.bpb, P.slot, 0};
    int mi = 0;
    if constexpr (MULTI) {
        const int rt = w0 / P.ngrp % P.rtiles;
        while (mi + 1 < mm.n && rt >= mm.mat[mi + 1].rt0) mi++;
        M = mm.mat[mi];
    }

    if (threadIdx.x == 0) {
        for (int i = 0; i < 3; i++) { mbar_init(&ctl->raw_full[i], P.tma ? 1 : MMQ_DQ_WARPS * 32); mbar_init(&ctl->raw_empty[i], MMQ_DQ_WARPS); }
        for (int i = 0; i < MMQ_A_MAX; i++) mbar_init(&ctl->a_ready[i], MMQ_DQ_WARPS);
        for (int i = 0; i < MMQ_B_NST; i++) { mbar_init(&ctl->b_full[i], 1); mbar_init(&ctl->step_done[i], 1); }
        mbar_init(&ctl->acc_ready, 1);
        mbar_init(&ctl->acc_free, MMQ_DQ_WARPS * CG);
        for (int i = 0; i < MMQ_B_NST; i++) mbar_init(&ctl->peer_ready[i], 1);
        ctl->abort = 0;
        mbar_fence_init();
    }
    if (warp == 0) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(P.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(P.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        pdl_trigger();   // behind the allocation: a later kernel's CTA on this SM must not take the columns first and wait for this one
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) mmq_cluster_sync();   // both CTAs' barriers are initialised before anything arrives on them from the other CTA
    tc_fence_after();
    const uint32_t tmem = *(volatile uint32_t *) &ctl->tmem_base;

    // Every role walks the same segments: unit w -> tile w / ngrp (token-tile group tile / rtiles, row tile tile % rtiles), K group w % ngrp.
    if (warp == 0 && rank != 0) {
        // ================= peer CTA of a pair: tell the leader when this CTA's stages of step g are filled =================
        if (lane == 0) {
            int g = 0;
            bool ok = true;
            for (int w = w0; w < w1 && ok;) {
                const int tile = w / P.ngrp, sbb = w - tile * P.ngrp, sbe = min(P.ngrp, sbb + (w1 - w));
                const int nsteps = min(4 * sbe, nstep_all) - 4 * sbb;
                for (int u = 0; u < nsteps; u++, g++) {
                    if (!mmq_wait(ctl, &ctl->b_full[g % P.b_nst], (g / P.b_nst) & 1)) { ok = false; break; }
                    if (!mmq_wait(ctl, &ctl->a_ready[g & amask], (g >> ashift) & 1)) { ok = false; break; }
                    mbar_arrive_cluster(&ctl->peer_ready[g % MMQ_B_NST], 0);
                }
                w += sbe - sbb;
            }
        }
        __syncwarp();
    } else if (warp == 0) {
        // ================= MMA issuer (the whole warp walks, an elected lane issues) =================
        int g = 0, seg = 0;                                      // CTA-wide step and segment counters (barrier phases follow them)
        bool ok = true;
        for (int w = w0; w < w1 && ok; seg++) {
            const int tile = w / P.ngrp, sbb = w - tile * P.ngrp, sbe = min(P.ngrp, sbb + (w1 - w));
            const int nacc = min(P.nacc, P.ttiles - (tile / P.rtiles) * P.nacc);
            const int nsteps = min(4 * sbe, nstep_all) - 4 * sbb;
            if (seg > 0 && !mmq_wait(ctl, &ctl->acc_free, (seg - 1) & 1)) break;   // the previous segment's accumulators have been read out
            tc_fence_after();
            for (int u = 0; u < nsteps; u++, g++) {
                const int sa = g & amask, sb = g % P.b_nst;
                if (!mmq_wait(ctl, &ctl->b_full[sb], (g / P.b_nst) & 1)) { ok = false; break; }
                if (!mmq_wait(ctl, &ctl->a_ready[sa], (g >> ashift) & 1)) { ok = false; break; }
                if (CG == 2 && !mmq_wait(ctl, &ctl->peer_ready[g % MMQ_B_NST], (g / MMQ_B_NST) & 1)) { ok = false; break; }
                tc_fence_after();
                const uint64_t da = umma_desc_sw128(smem_u32(a_st + (size_t) sa * MMQ_A_BYTES));
                const uint64_t db = umma_desc_sw128(smem_u32(b_st + (size_t) sb * b_bytes));
                const uint64_t db2 = umma_desc_sw128(smem_u32(b_st + (size_t) sb * b_bytes + b1c));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < MMQ_BK / 16; k++) {
                        if (CG == 2) {
                            umma_f16_cg2(tmem, da + 2 * k, db + 2 * k, P.idesc, (u | k) != 0);
                            if (nacc == 2) umma_f16_cg2(tmem + 256, da + 2 * k, db2 + 2 * k, P.idesc, (u | k) != 0);
                        } else {
                            umma_f16(tmem, da + 2 * k, db + 2 * k, P.idesc, (u | k) != 0);
                            if (nacc == 2) umma_f16(tmem + 256, da + 2 * k, db2 + 2 * k, P.idesc, (u | k) != 0);
                        }
                    }
                    if (CG == 2) umma_commit_cg2(&ctl->step_done[g % MMQ_B_NST]); else umma_commit(&ctl->step_done[g % MMQ_B_NST]);
                }
                __syncwarp();
            }
            if (elect_one()) {
                if (CG == 2) umma_commit_cg2(&ctl->acc_ready); else umma_commit(&ctl->acc_ready);
            }
            __syncwarp();
            w += sbe - sbb;
        }
    } else if (warp == 1) {
        // ================= activation producer: runs up to b_nst steps ahead of the tensor core =================
        pdl_wait();                // activations are the kernel in front's; weights are fetched and expanded meanwhile
        const size_t tile_stride = (size_t) nstep_all * b1;
        int g = 0;
        bool ok = true;
        for (int w = w0; w < w1 && ok;) {
            const int tile = w / P.ngrp, sbb = w - tile * P.ngrp, sbe = min(P.ngrp, sbb + (w1 - w));
            const int tt0 = (tile / P.rtiles) * P.nacc;
            const int nacc = min(P.nacc, P.ttiles - tt0);
            const int nsteps = min(4 * sbe, nstep_all) - 4 * sbb;
            const uint8_t * Bt = P.B + (size_t) tt0 * tile_stride + (size_t) sbb * 4 * b1 + (size_t) rank * b1c;
            for (int u = 0; u < nsteps; u++, g++) {
                const int sb = g % P.b_nst;
                if (g >= P.b_nst) {   // step g - b_nst consumed this stage
                    const int f = g - P.b_nst;
                    if (!mmq_wait(ctl, &ctl->step_done[f % MMQ_B_NST], (f / MMQ_B_NST) & 1)) { ok = false; break; }
                }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&ctl->b_full[sb], (uint32_t) (nacc * b1c));
                    for (int a = 0; a < nacc; a++)
                        bulk_g2s_plain(b_st + (size_t) sb * b_bytes + (size_t) a * b1c, Bt + (size_t) a * tile_stride + (size_t) u * b1, (uint32_t) b1c, &ctl->b_full[sb]);
                }
                __syncwarp();
            }
            w += sbe - sbb;
        }
    } else if (warp == MMQ_RAW_WARP) {
        // ================= raw blocks: a K group of the tile's rows is one box, up to nraw groups ahead =================
        if (P.tma) {
            const int nx = w1 - w0;
            int sb = w0 % P.ngrp, rt = w0 / P.ngrp % P.rtiles, slot = 0, ph = 1;
            for (int x = 0; x < nx; x++) {
                if (x >= P.nraw && !mmq_wait(ctl, &ctl->raw_empty[slot], ph)) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&ctl->raw_full[slot], (uint32_t) (MMQ_BM * M.slot));
                    tma_raw(smem_u32(raw + (size_t) slot * MMQ_BM * P.slot), &mm.map[mi], (sb * M.bpb & ~15) >> 1, ((rt - M.rt0) * CG + (int) rank) * MMQ_BM, smem_u32(&ctl->raw_full[slot]));
                }
                __syncwarp();
                if (++slot == P.nraw) { slot = 0; ph ^= 1; }
                if (++sb == P.ngrp) { sb = 0; if (++rt == P.rtiles) rt = 0; }
            }
        }
    } else {
        // ================= weight expansion =================
        const int dt = threadIdx.x - MMQ_DQ_WARP0 * 32;        // 0..511
        const int r = dt >> 2, h = (dt >> 1) & 1, hh = dt & 1;
        bool ok = true;
        // this thread fetches its own half of the row's block: 16-byte cp.async pieces of the 16-B aligned window around it
        const int64_t lim = (M.total_bytes + 15) & ~(int64_t) 15;
        const int cpr = M.slot >> 4, p_lo = cpr * (dt & 3) / 4, p_hi = cpr * ((dt & 3) + 1) / 4;   // this thread's quarter of the row's window
        const int nx = w1 - w0;                                 // groups this CTA walks, x = 0 .. nx-1 across its segments
        // fetch cursor: the group nraw-1 ahead of the one being expanded (tile / K group tracked incrementally: no divisions in the loop)
        int f_x = 0, f_sb, f_rt;
        { const int tile = w0 / P.ngrp; f_sb = w0 - tile * P.ngrp; f_rt = tile % P.rtiles; }
        auto fetch_next = [&](int slot) {                       // issues group f_x of this CTA into raw slot `slot`, advances the cursor
            const int gr = min((f_rt * CG + (int) rank) * MMQ_BM + r, M.N - 1);   // never with several matrices: those come by boxes
            const int64_t src0 = ((int64_t) gr * M.row_bytes + (int64_t) f_sb * M.bpb) & ~(int64_t) 15;
            uint8_t * dst0 = raw + ((size_t) slot * MMQ_BM + r) * P.slot;
            for (int pc = p_lo; pc < p_hi; pc++)
                if (src0 + pc * 16 + 16 <= lim) cp_async16(dst0 + pc * 16, M.W + src0 + pc * 16);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&ctl->raw_full[slot])) : "memory");
            f_x++;
            if (++f_sb == P.ngrp) { f_sb = 0; if (++f_rt == P.rtiles) f_rt = 0; }
        };
        if (!P.tma) for (int i = 0; i < P.nraw - 1 && i < nx; i++) fetch_next(i);
        // the four 16-byte pieces this thread writes per step, already swizzled
        const uint32_t arow = r * 128;
        const uint32_t o0 = arow + (((4 * h + 2 * hh + 0) ^ (r & 7)) << 4), o1 = arow + (((4 * h + 2 * hh + 1) ^ (r & 7)) << 4);
        int g = 0, seg = 0;
        int rs = 0, rph = 0;                                    // raw slot / phase of the group being expanded
        int prs = P.nraw - 1, pph = 1;                          // ... of the group before it (the slot the next fetch goes into)
        for (int w = w0; w < w1 && ok; seg++) {
            const int tile = w / P.ngrp, sbb = w - tile * P.ngrp, sbe = min(P.ngrp, sbb + (w1 - w));
            const int row0 = ((tile % P.rtiles - M.rt0) * CG + (int) rank) * MMQ_BM;
            const int gr = min(row0 + r, M.N - 1);
            for (int sb = sbb; sb < sbe && ok; sb++) {
                // refill the slot the previous group used, once every expansion warp has left it
                if (!P.tma && f_x < nx) {
                    if (f_x >= P.nraw && !mmq_wait(ctl, &ctl->raw_empty[prs], pph)) { ok = false; break; }
                    fetch_next(prs);
                }
                if (!mmq_wait(ctl, &ctl->raw_full[rs], rph)) { ok = false; break; }
                const int64_t g0 = (int64_t) gr * M.row_bytes + (int64_t) sb * M.bpb;
                const uint8_t * blk = raw + (size_t) rs * MMQ_BM * P.slot + (size_t) r * M.slot + (g0 & 15);
                const int nst = min(4, nstep_all - 4 * sb);      // the last group of a K % 256 != 0 row (32-element block types) is short
                constexpr bool K45 = TYPE == T_Q4_K || TYPE == T_Q5_K;
                const bool second = MIXED && M.second;           // Q6_K beside Q4_K or Q5_K
                KGroup<TYPE> kg;
                if constexpr (K45) {
                    if (!second) {
                        kg.load(blk, h, hh);
                        kg.loaded();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&ctl->raw_empty[rs]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c >= nst) break;
                    uint32_t v[8];
                    if constexpr (MIXED) {
                        if (second) expand<TYPE2>(blk, c, h, hh, v);
                        else kg.expand(c, h, v);
                    } else if constexpr (K45) kg.expand(c, h, v);
                    else expand<TYPE>(blk, c, h, hh, v);
                    if (g >= P.a_nst) {     // step g - a_nst has consumed this A stage
                        const int f = g - P.a_nst;
                        if (!mmq_wait(ctl, &ctl->step_done[f % MMQ_B_NST], (f / MMQ_B_NST) & 1)) { ok = false; break; }
                    }
                    uint8_t * as = a_st + (size_t) (g & amask) * MMQ_A_BYTES;
                    *reinterpret_cast<uint4 *>(as + o0) = make_uint4(v[0], v[1], v[2], v[3]);
                    *reinterpret_cast<uint4 *>(as + o1) = make_uint4(v[4], v[5], v[6], v[7]);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy stores -> visible to the tensor core's async proxy
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctl->a_ready[g & amask]);
                    g++;
                }
                if (!K45 || second) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctl->raw_empty[rs]);
                }
                prs = rs; pph = rph;
                if (++rs == P.nraw) { rs = 0; rph ^= 1; }
            }
            pdl_wait();            // residuals are read and results written behind it
            if constexpr (CUT) {
                // ================= epilogue of a part: partial sums [token][row] go over the stages' memory (every load and MMA of this CTA is done),
                // one accumulator after the other; token t is added up, in the parts' order, by CTA t % parts =================
                const bool acc_ok = ok && mmq_wait(ctl, &ctl->acc_ready, 0);
                tc_fence_after();
                const int tt0 = (tile / P.rtiles) * P.nacc, nacc = min(P.nacc, P.ttiles - tt0);
                const int quad = warp & 3, grp = (warp - MMQ_DQ_WARP0) >> 2, n = row0 + quad * 32 + lane;
                float * red = reinterpret_cast<float *>(smem) + quad * 32 + lane;
                const float bias = (M.bias && n < M.N) ? M.bias[n] : 0.f;
                for (int a = 0; a < nacc; a++) {
                    const int t0 = (tt0 + a) * BN, tn = min(BN, P.T - t0);
                    for (int c0 = 16 * grp; c0 < tn && acc_ok; c0 += 64) {
                        uint32_t v[16];
                        const uint32_t taddr = tmem + ((uint32_t) (quad * 32) << 16) + (uint32_t) (a * 256 + c0);
                        asm volatile(
                            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                              "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                            : "r"(taddr)
                            : "memory");
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 16; i++) red[(c0 + i) * MMQ_BM] = __uint_as_float(v[i]);
                    }
                    __syncwarp();
                    mmq_cluster_sync();
                    if (n < M.N) {
                        constexpr int U = 8;                     // tokens of a thread at once, two parts of them on their way: what takes time is the latency
                        const int step = 4 * P.parts;
                        for (int t = part + P.parts * grp; t < tn; t += U * step) {
                            float sum[U], f[2][U];                // bias and residual ride on part 0
#pragma unroll
                            for (int i = 0; i < U; i++) sum[i] = P.resid && t + i * step < tn ? P.resid[(size_t) (t0 + t + i * step) * (size_t) M.N + n] : 0.f;
                            for (int c = 0; c < P.parts; c += 2) {
#pragma unroll
                                for (int h = 0; h < 2; h++)
                                    if (c + h < P.parts) {
                                        const uint32_t at = mmq_peer_addr(smem_u32(red + t * MMQ_BM), (uint32_t) (c + h));
#pragma unroll
                                        for (int i = 0; i < U; i++)
                                            if (t + i * step < tn) f[h][i] = mmq_peer_f32(at + (uint32_t) (i * step * MMQ_BM * 4));
                                    }
#pragma unroll
                                for (int h = 0; h < 2; h++)
                                    if (c + h < P.parts) {
#pragma unroll
                                        for (int i = 0; i < U; i++) sum[i] = c + h == 0 ? __fadd_rn(__fadd_rn(f[h][i], bias), sum[i]) : __fadd_rn(sum[i], f[h][i]);
                                    }
                            }
#pragma unroll
                            for (int i = 0; i < U; i++)
                                if (t + i * step < tn) M.dst[(size_t) (t0 + t + i * step) * (size_t) M.N + n] = sum[i];
                        }
                    }
                    __syncwarp();
                    mmq_cluster_read();   // read by every CTA: the next accumulator may go there, or the CTA leave
                }
            } else
            // ================= epilogue of the segment: four consecutive warps cover the four 32-lane quadrants of TMEM =================
            // All 16 expansion warps read out: a warp may only read quadrant warp % 4, its group (warp - 2) / 4 takes every fourth chunk of 16
            // columns.  Chunk ch holds tokens tt0 * BN + 16 ch ..: two accumulators lie 256 columns apart and are only used with BN = 256.
            // What bounds it is instruction issue (128 x 512 values; 8 warps with a 64-bit index product, two tests and a select per value
            // took 20 of the 26 us that a segment cost beyond its MMA steps), hence the walking pointers and the paths without residual tests.
            {
                const bool acc_ok = ok && mmq_wait(ctl, &ctl->acc_ready, seg & 1);
                tc_fence_after();
                const int tt0 = (tile / P.rtiles) * P.nacc;
                const int nch = min(P.nacc, P.ttiles - tt0) * (BN >> 4);
                const bool first = sbb == 0, whole = first && sbe == P.ngrp;   // bias / residual ride on the K group 0 segment
                const int quad = warp & 3;
                const int n = row0 + quad * 32 + lane;
                const bool live = acc_ok && n < M.N;
                const float bias = (M.bias && live && first) ? M.bias[n] : 0.f;
                const float * rp = (P.resid && first && live) ? P.resid + n : nullptr;
                const size_t ldd = (size_t) M.N;
                for (int ch = (warp - MMQ_DQ_WARP0) >> 2; ch < nch; ch += 4) {
                    const int t0 = tt0 * BN + ch * 16;
                    const int nt = min(16, P.T - t0);            // tokens of the chunk (<= 0: padding only)
                    if (nt <= 0) break;
                    float y[16];
                    // all 16 residual loads in flight at once, ahead of the stores they could alias as far as the compiler knows
                    if (rp) {
                        const float * q = rp + (size_t) t0 * ldd;
#pragma unroll
                        for (int i = 0; i < 16; i++) y[i] = i < nt ? q[i * ldd] : 0.f;
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; i++) y[i] = 0.f;
                    }
                    __syncwarp();
                    uint32_t v[16];
                    const uint32_t taddr = tmem + ((uint32_t) (quad * 32) << 16) + (uint32_t) (ch * 16);
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                        : "r"(taddr)
                        : "memory");
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (live) {
                        float * d = M.dst + (size_t) t0 * ldd + n;
#pragma unroll
                        for (int i = 0; i < 16; i++) y[i] = __fadd_rn(__fadd_rn(__uint_as_float(v[i]), bias), y[i]);
                        if (whole && nt == 16) {
#pragma unroll
                            for (int i = 0; i < 16; i++, d += ldd) *d = y[i];
                        } else if (whole) {
#pragma unroll
                            for (int i = 0; i < 16; i++, d += ldd) if (i < nt) *d = y[i];
                        } else if (nt == 16) {
#pragma unroll
                            for (int i = 0; i < 16; i++, d += ldd) atomicAdd(d, y[i]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 16; i++, d += ldd) if (i < nt) atomicAdd(d, y[i]);
                        }
                    }
                    __syncwarp();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {                                 // the issuer (of the leader CTA) may overwrite the accumulators
                    if (CG == 2) mbar_arrive_cluster(&ctl->acc_free, 0); else mbar_arrive(&ctl->acc_free);
                }
            }
            w += sbe - sbb;
        }
    }
    if (CUT && (warp < MMQ_DQ_WARP0 || warp == MMQ_RAW_WARP)) {   // the cluster's barriers count every warp
        const int rounds = min(P.nacc, P.ttiles - (w0 / P.ngrp / P.rtiles) * P.nacc);
        for (int i = 0; i < rounds; i++) { mmq_cluster_sync(); mmq_cluster_read(); }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) mmq_cluster_sync();   // the pair leaves together: the leader's MMAs and commits reach into the peer's shared memory
    if (warp == 0) {
        tc_fence_after();
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P.tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P.tmem_cols) : "memory");
    }
}

// ---- activation rows -> q8_K (exactly as the CPU backend quantizes them) -> fp16, written in the tiled UMMA image ----
// blk32: the weight type is Q8_0 / Q5_1, whose CPU dot quantizes the activation per 32 values (q8_0 / q8_1: d = amax / 127 stored
// as f16, q = round-half-even(x * 127 / amax), quantize_row_q8_0 ggml-quants.c:943-1010) instead of per 256 (q8_K).
// Fused producers of the activation (pre_kind): 1 = silu(x) * aux[t][k] (llm_build_ffn's SILU + MUL in front of ffn_down, the f32 product never
// goes to HBM), 2 = rms_norm(x) * aux[k] (llm_build_norm in front of q|k|v and gate|up): the same arithmetic, rounding for rounding, as
// k_silu_mul / k_rms_norm_rows followed by the plain pass.
// Bound by the latency of its loads: a warp's first two blocks are fetched ahead of the norm's sum, which loads eight at a time, and long rows go over two CTAs
// (a prompt of 512 tokens and 4 layers of 4096 / 14336: 1632 -> 1561 us with it).
__device__ __forceinline__ float mmq_silu(float x) { return __fdiv_rn(x, 1.0f + expf(-x)); }   // ggml.c:2560
__global__ void __launch_bounds__(256) k_mmq_prep(const float * x, int64_t ldx, int T, int K, int BN, uint8_t * out,
                                                  int blk32, int pre_kind, const float * aux, int64_t ld_aux, float eps) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nblk = (K + 255) / 256;
    const int t = blockIdx.x;                       // 0 .. Tpad-1
    const int b_bytes = BN * 128;
    float nscale = 1.f;
    pdl_trigger();
    pdl_wait();
    // a warp's blocks two at a time, eight warps and gridDim.y CTAs apart; the first two are on their way while the row's norm is taken
    const int step = 8 * (int) gridDim.y;
    float4 xa[2], xb[2];
    auto fetch = [&](int b0) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int b = b0 + j * step;
            const float4 * p = reinterpret_cast<const float4 *>(x + (size_t) t * ldx + (size_t) b * 256 + lane * 8);
            const bool live = t < T && b < nblk && b * 256 + lane * 8 < K;   // K % 32 == 0: a 4-lane group (one 32-block) is live or dead as a whole
            xa[j] = live ? p[0] : make_float4(0.f, 0.f, 0.f, 0.f);
            xb[j] = live ? p[1] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    const int first = warp + 8 * (int) blockIdx.y;
    fetch(first);
    if (pre_kind == 2 && t < T) {                   // k_rms_norm_rows' sum, in its order (ggml.c:11950-11996: double-precision sum of squares)
        __shared__ double red[8];
        __shared__ float s_scale;
        const float * xr = x + (size_t) t * ldx;
        double sum = 0.0;
#pragma unroll 8
        for (int i = threadIdx.x; i < K; i += 256) sum += (double) __fmul_rn(xr[i], xr[i]);
        sum = warp_sum_d(sum);
        if (lane == 0) red[warp] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            double tt = 0;
            for (int i = 0; i < 8; i++) tt += red[i];
            const float mean = (float) (tt / (double) K);
            s_scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
        }
        __syncthreads();
        nscale = s_scale;
    }
    for (int b0 = first; b0 < nblk; b0 += 2 * step) {
        if (b0 != first) fetch(b0);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int b = b0 + u * step;
            if (b >= nblk) break;
            const bool live = b * 256 + lane * 8 < K;
            float v[8] = {xa[u].x, xa[u].y, xa[u].z, xa[u].w, xb[u].x, xb[u].y, xb[u].z, xb[u].w};
            if (pre_kind && t < T && live) {
                const float4 * q = reinterpret_cast<const float4 *>(aux + (pre_kind == 1 ? (size_t) t * ld_aux : (size_t) 0) + (size_t) b * 256 + lane * 8);
                const float4 e = q[0], f = q[1];
                const float w[8] = {e.x, e.y, e.z, e.w, f.x, f.y, f.z, f.w};
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = pre_kind == 1 ? __fmul_rn(mmq_silu(v[i]), w[i]) : __fmul_rn(__fmul_rn(v[i], nscale), w[i]);
            }
            float amax = 0.f, vmax = 0.f;
            int idx = 0x7fffffff;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float ax = fabsf(v[i]);
                if (ax > amax) { amax = ax; vmax = v[i]; idx = lane * 8 + i; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float oa = __shfl_xor_sync(0xffffffffu, amax, o);
                const float ov = __shfl_xor_sync(0xffffffffu, vmax, o);
                const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
                if (oa > amax || (oa == amax && oi < idx)) { amax = oa; vmax = ov; idx = oi; }
            }
            uint32_t h[4] = {0u, 0u, 0u, 0u};
            if (blk32) {
                float am = 0.f;
#pragma unroll
                for (int i = 0; i < 8; i++) am = fmaxf(am, fabsf(v[i]));
                am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
                am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
                const float d = __half2float(__float2half_rn(__fdiv_rn(am, 127.f)));
                const float id = am != 0.f ? __fdiv_rn(127.f, am) : 0.f;
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; i++) f[i] = __fmul_rn(d, (float) __float2int_rn(__fmul_rn(v[i], id)));
                h[0] = pack_h2(f[0], f[2]); h[1] = pack_h2(f[1], f[3]); h[2] = pack_h2(f[4], f[6]); h[3] = pack_h2(f[5], f[7]);
            } else if (amax != 0.f) {
                const float iscale = __fdiv_rn(-127.f, vmax);
                const float d = __fdiv_rn(1.f, iscale);
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    int q = nearest_int_magic(__fmul_rn(iscale, v[i]));
                    q = q < 127 ? q : 127;
                    f[i] = __fmul_rn(d, (float) q);
                }
#pragma unroll
                // within every 4 consecutive k the order is (0,2,1,3): the weight expansion produces its half2 pairs that way
                h[0] = pack_h2(f[0], f[2]); h[1] = pack_h2(f[1], f[3]); h[2] = pack_h2(f[4], f[6]); h[3] = pack_h2(f[5], f[7]);
            }
            const int k = b * 256 + lane * 8;
            const int kc = k >> 6, j = (k & 63) >> 3;
            const int tt = t / BN, tl = t % BN;
            uint8_t * dstp = out + ((size_t) tt * (K / 64) + kc) * b_bytes + (size_t) tl * 128 + (size_t) ((j ^ (tl & 7)) << 4);
            if (live) *reinterpret_cast<uint4 *>(dstp) = make_uint4(h[0], h[1], h[2], h[3]);
        }
    }
}

static int mmq_pick_bn(int T) {
    if (T >= 256) return 256;
    int bn = (T + 15) / 16 * 16;
    return bn < 16 ? 16 : bn;
}
size_t mmq_workspace_bytes(int64_t K, int64_t T) {
    const int BN = mmq_pick_bn((int) T);
    const int64_t tpad = (T + BN - 1) / BN * BN;
    return (size_t) (tpad * K * 2);
}
bool mmq_supported(int type, int64_t K) {
    if (is_kquant(type)) return K % 256 == 0 && K >= 256;
    return (type == T_Q8_0 || type == T_Q5_1) && K % 64 == 0 && K >= 256;   // 32-element blocks: two per 64-element step
}

template <int TYPE, int CG, bool CUT, int TYPE2 = 0>
static cudaError_t mmq_launch_typed2(const MmqParams & P, const MmqMats<(TYPE2 > 0)> & mats, dim3 grid, size_t smem, cudaStream_t st, bool pdl) {
    static FuncAttrCache attr_cache;
    cudaError_t e = ensure_dyn_smem(attr_cache, (const void *) k_mmq_tc<TYPE, CG, CUT, TYPE2>, smem, false);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(MMQ_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CUT ? (unsigned) P.parts : CG; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CG > 1 || CUT ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_mmq_tc<TYPE, CG, CUT, TYPE2>, P, mats);
}
template <int TYPE>
static cudaError_t mmq_launch_typed(const MmqParams & P, const MmqMats<false> & map_w, int cg, dim3 grid, size_t smem, cudaStream_t st, bool pdl) {
    if (P.parts > 1) return mmq_launch_typed2<TYPE, 1, true>(P, map_w, grid, smem, st, pdl);
    return cg == 2 ? mmq_launch_typed2<TYPE, 2, false>(P, map_w, grid, smem, st, pdl) : mmq_launch_typed2<TYPE, 1, false>(P, map_w, grid, smem, st, pdl);
}
// Clusters of `parts` CTAs of this kernel that run at the same time (a CTA takes an SM; a cluster stays within a group of SMs): what
// cudaOccupancyMaxActiveClusters says on a B200, 5 and 7 from below.  A table and no query, so that the order of a sum does not follow which SMs of a GPU
// are there; where fewer clusters fit, the rest of them come after.
static int mmq_clusters(int parts, int nsm) {
    constexpr int of_148[MMQ_MAX_PARTS + 1] = {0, 148, 74, 45, 33, 24, 22, 16, 15};
    return of_148[parts] * nsm / 148;
}

// How a launch's tiles are shared:
//   parts > 1   the CTAs of a cluster cut one tile's K into equal consecutive parts and add their sums in the parts' order through distributed shared
//               memory
//   chain > 0   chains of tiles, each in equal contiguous shares for one CTA more than it has tiles: every tile is cut once
//   else        contiguous shares of upc units: whole tiles, or at least a tile less one group, so that again no tile is cut twice
// Where a tile is cut once its two sums meet on a cleared output: in either order they give the same bits.  An element's sum so has one order,
// fixed by the launch's tiles and K groups, not by its tokens: the same call gives the same bits, and k-quant weights give a row the same
// bits with 8 or 511 others beside it.
// Costs in us on B200, Q4_K, 512 tokens: a unit 3.05 (2.3 with few tokens: the chain of a step), a segment's fill and read-out 8, the join of
// p parts 7.5 + 1.25 p (what distributed shared memory gives: 256 KB a CTA; in proportion to the tokens), the clearing pass 3 + bytes /
// 6.2 TB/s.  Measured with the activation pass, K = 4096, 512 tokens: 1024 rows whole 63.5, 2 parts 48.7, 4 parts 38.4, 8 parts 34.1; 4096 rows
// whole 63.7, 4 parts 37.2; 64 tokens: 1024 rows 53.3, 31.9, 21.8, 16.6.  8192 x 8192 in halves: 79.1 by a cluster, 74 onto a cleared
// output; 64 tokens 56 and 57.  20480 x 2048: whole tiles 71.4, shares of 9 units 58.4.
// What the order costs: shares for every SM whose sums meet as they arrive took (512 / 64 tokens, then -> now) 20.0 / 11.9 -> 34.1 / 16.6 at
// 1024 x 4096, 31.4 / 21.0 -> 37.2 / 21.9 at 4096 x 4096, 25.1 / 14.8 -> 32.4 / 18.8 at 3072 x 3072, 74.0 / 54.9 -> 78.3 / 55.1 at 4096 x 14336,
// 229 / 169 -> 244 / 183 at 8192 x 28672, 175 / 126 -> 183 / 138 at 12800 x 14336; 37.8 / 29.7 -> 28.9 / 19.9 at 2048 x 2048, where tiles stayed whole.
struct MmqCut { int parts, chain, upc; double us; };
static int64_t mmq_chain_ctas(int64_t tiles, int m) { return tiles / m * (m + 1) + (tiles % m ? tiles % m + 1 : 0); }
static MmqCut mmq_pick_cut(int64_t tiles, int ngrp, int nsm, int max_parts, double tokens) {
    const double unit = 3.05, seg = 8.0, tile_us = 128.0 * 512.0 * 4.0 / 6.2e6, clear = 3.0 + (double) tiles * tile_us;
    const int rounds = (int) ((tiles + nsm - 1) / nsm);
    MmqCut best{1, 0, rounds * ngrp, 0.0};
    double best_us = rounds * (ngrp * unit + seg);
    auto consider = [&](const MmqCut & c, double us) { if (us < best_us) { best_us = us; best = c; } };
    const int upc = std::max((int) ((tiles * ngrp + nsm - 1) / nsm), ngrp - 1);
    if (upc % ngrp != 0) consider({1, 0, upc, 0.0}, upc * unit + ((upc + ngrp - 2) / ngrp + 1) * seg + clear);
    for (int m = 2; m <= 8; m++)
        if (mmq_chain_ctas(tiles, m) <= nsm) consider({1, m, 0, 0.0}, (m * ngrp + m) / (m + 1) * unit + 2 * seg + clear);
    // two halves: by a cluster or a chain of one tile, whichever is the faster one for these tokens; the bits are the same
    const bool pairs = max_parts >= 2 && tiles <= mmq_clusters(2, nsm);
    if (tiles * 2 <= nsm && ngrp >= 2)
        consider(pairs && 10.0 * tokens <= 3.0 * 512.0 + (double) tiles * tile_us * tokens ? MmqCut{2, 0, 0, 0.0} : MmqCut{1, 1, 0, 0.0}, (ngrp + 1) / 2 * unit + seg + std::min(10.0, clear));
    for (int p = 3; p <= max_parts && p <= ngrp && tiles * p <= nsm; p++) {
        const double us = (ngrp + p - 1) / p * unit + seg + 7.5 + 1.25 * p;
        if (us < best_us && tiles <= mmq_clusters(p, nsm)) consider({p, 0, 0, 0.0}, us);
    }
    best.us = best_us;
    return best;
}

// bytes of one 256-K group of a row, and the 16-byte aligned window reserved for it (Q6_K and Q8_0 rows are not 16-B aligned)
static int mmq_group_bytes(int type) { return type == T_Q4_K ? BYTES_Q4_K : type == T_Q5_K ? BYTES_Q5_K : type == T_Q6_K ? BYTES_Q6_K : type == T_Q8_0 ? 8 * BYTES_Q8_0 : 8 * BYTES_Q5_1; }
static int mmq_slot_bytes(int type) { return type == T_Q6_K ? 240 : type == T_Q8_0 ? 288 : mmq_group_bytes(type); }
// the raw blocks of a matrix by boxes; false: its rows do not lie at multiples of 16 bytes
static bool mmq_map(CUtensorMap & map, int type, const void * W, int64_t N, int64_t K) {
    const int64_t row = row_bytes(type, K);
    const EncodeTiled fn = row % 16 == 0 && ((uintptr_t) W & 15) == 0 ? encode_tiled() : nullptr;
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t) row / 2, (cuuint64_t) N}, strides[1] = {(cuuint64_t) row};   // 16-bit entries: a box is at most 256 of them wide
    const cuuint32_t box[2] = {(cuuint32_t) mmq_slot_bytes(type) / 2, MMQ_BM}, one[2] = {1, 1};
    return fn(&map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, (void *) W, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
static cudaError_t mmq_prepare(int type, const float * x, int64_t ldx, int64_t T, int64_t K, int BN, void * ws, const MmqPre * pre, bool pdl, cudaStream_t st) {
    const int kind = pre ? pre->kind : 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned) ((T + BN - 1) / BN * BN), kind != 2 && K >= 32 * 256 ? 2 : 1);   // long rows over two CTAs (a norm wants the whole row)
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_mmq_prep, x, ldx, (int) T, (int) K, BN, (uint8_t *) ws, is_kquant(type) ? 0 : 1, kind, pre ? pre->aux : (const float *) nullptr,
                              pre ? pre->ld_aux : (int64_t) 0, pre ? pre->eps : 0.f);
}
// P's tensor memory, instruction and ring depths; returns the shared memory, 0: more than there is.  3 raw super-block slots (HBM latency) if they fit, and as many
// activation stages (2..4) as the 227 KB budget leaves; 4 expanded-weight stages when a CTA pair halves the activation stages (the handshake "MMA
// done -> store the next tile -> MMA" then has three MMA steps of slack instead of one), else 2
static size_t mmq_rings(MmqParams & P, int cg) {
    uint32_t cols = 32;
    while ((int) cols < P.BN) cols <<= 1;
    P.tmem_cols = P.nacc == 2 ? 512 : cols;
    // kind::f16 instruction descriptor (cute/arch/mma_sm100_desc.hpp InstrDescriptor): D=f32, A=B=f16, both K-major, N>>3, M>>4
    P.idesc = (1u << 4) | ((uint32_t) (P.BN >> 3) << 17) | ((uint32_t) ((MMQ_BM * cg) >> 4) << 24);
    auto smem_for = [&](int nraw, int b_nst) {
        return 1024 + (size_t) P.a_nst * MMQ_A_BYTES + (size_t) b_nst * P.nacc * (P.BN / cg) * 128 + (size_t) nraw * MMQ_BM * P.slot + MMQ_CTL_BYTES;
    };
    static const int force_a = getenv("PB200_MMQ_A_NST") ? atoi(getenv("PB200_MMQ_A_NST")) : 0;
    P.a_nst = force_a == 2 || force_a == 4 ? force_a : (cg == 2 ? 4 : 2);
    P.nraw = 3;
    if (smem_for(3, 2) > 232448) P.nraw = 2;
    if (smem_for(P.nraw, 2) > 232448) P.a_nst = 2;
    P.b_nst = MMQ_B_NST;
    while (P.b_nst > 2 && smem_for(P.nraw, P.b_nst) > 232448) P.b_nst--;
    const size_t smem = smem_for(P.nraw, P.b_nst);
    return smem > 232448 ? 0 : smem;
}

cudaError_t launch_mmq(int type, const void * W, int64_t N, int64_t K, const float * x, int64_t ldx, int64_t T, float * dst, const float * bias,
                       const float * resid, void * ws, cudaStream_t st, bool reuse_prep, const MmqPre * pre, bool pdl) {
    if (pre && pre->kind != 0 && (!pre->aux || K % 256 != 0 || pre->kind < 0 || pre->kind > 2)) return cudaErrorInvalidValue;
    if (!mmq_supported(type, K) || N <= 0 || T <= 0) return cudaErrorInvalidValue;
    const int BN = mmq_pick_bn((int) T);
    const int tpad = (int) ((T + BN - 1) / BN * BN);

    MmqParams P{};
    P.abort_flag = abort_flag();
    P.W = (const uint8_t *) W;
    P.B = (const uint8_t *) ws;
    P.dst = dst;
    P.bias = bias;
    P.resid = resid;
    P.row_bytes = row_bytes(type, K);
    P.total_bytes = P.row_bytes * N;
    P.N = (int) N;
    P.K = (int) K;
    P.T = (int) T;
    P.BN = BN;
    P.bpb = mmq_group_bytes(type);
    P.slot = mmq_slot_bytes(type);
    P.ttiles = tpad / BN;
    // CTA pairs (tcgen05 cta_group::2, PB200_MMQ_CG=2): two row tiles form one M = 256 MMA, each CTA stages only half of the activation tile
    // (L2 -> SM traffic halves, room for 4 expanded-weight stages).  Built and measured: parity green, but 5-7 % SLOWER than one CTA per
    // MMA at every shape (profiles/r2_mmq_probe.txt) — neither the activation ring nor the weight-stage depth was the limiter, the
    // weight-expansion warps were (8 -> 16 warps: +19 %).  The single-CTA form is the default.
    static const int force_cg = getenv("PB200_MMQ_CG") ? atoi(getenv("PB200_MMQ_CG")) : 0;
    const int rt1 = (int) ((N + MMQ_BM - 1) / MMQ_BM);
    const int cg = (force_cg == 2 && rt1 >= 2 && BN % 32 == 0) ? 2 : 1;
    P.rtiles = (rt1 + cg - 1) / cg;            // row-tile groups (pairs)
    // two accumulators per output tile halve the weight-expansion work per FLOP (measured 1040 vs 590 TFLOP/s at full occupancy)
    static const int force_nacc = getenv("PB200_MMQ_NACC") ? atoi(getenv("PB200_MMQ_NACC")) : 0;
    P.nacc = (P.ttiles >= 2 && force_nacc != 1) ? 2 : 1;
    // ... if the shared-memory budget allows it: Q8_0's 288-byte raw slots leave no room for two 64-KB activation stages
    if (P.nacc == 2 && 1024 + (size_t) 2 * MMQ_A_BYTES + (size_t) 2 * 2 * (BN / cg) * 128 + (size_t) 2 * MMQ_BM * P.slot + MMQ_CTL_BYTES > 232448) P.nacc = 1;
    const int tgroups = (P.ttiles + P.nacc - 1) / P.nacc;
    P.ngrp = (int) ((K / MMQ_BK + 3) / 4);
    static const bool whole_tiles = getenv("PB200_MMQ_WHOLE_TILES") != nullptr;   // A/B: one tile per CTA (no split, no atomics)
    const int64_t tiles = (int64_t) P.rtiles * tgroups, total = tiles * P.ngrp;
    if (total > 0x7fffffff) return cudaErrorInvalidValue;
    P.total_units = (int) total;
    if (!reuse_prep) {
        const cudaError_t e0 = mmq_prepare(type, x, ldx, T, K, BN, ws, pre, pdl, st);
        if (e0 != cudaSuccess) return e0;
    }
    const size_t smem = mmq_rings(P, cg);
    if (smem == 0) return cudaErrorInvalidConfiguration;
    const int nsm = sm_count() / cg;           // CTAs (pairs) that can be resident: one CTA per SM
    MmqCut cut = mmq_pick_cut(tiles, P.ngrp, nsm, cg == 1 && (size_t) MMQ_BM * BN * 4 <= smem - 1024 - MMQ_CTL_BYTES ? MMQ_MAX_PARTS : 1, (double) std::min<int64_t>(T, 512));
    if (whole_tiles) cut = {1, 0, P.ngrp, 0.0};
    P.parts = cut.parts;
    P.chain = cut.chain;
    P.upc = cut.upc;
    if (cut.chain > 0 || (cut.parts == 1 && cut.upc % P.ngrp != 0)) {   // some tile is shared by two CTAs: their sums meet in dst by atomic add
        cudaError_t e0 = cudaMemsetAsync(dst, 0, (size_t) T * (size_t) N * sizeof(float), st);
        if (e0 != cudaSuccess) return e0;
    }
    MmqMats<false> map_w{};
    P.tma = mmq_map(map_w.map[0], type, W, N, K);
    dim3 grid((unsigned) (cut.parts > 1 ? tiles * cut.parts : cg * (cut.chain > 0 ? mmq_chain_ctas(tiles, cut.chain) : (total + cut.upc - 1) / cut.upc)), 1, 1);
    if (type == T_Q4_K) return mmq_launch_typed<T_Q4_K>(P, map_w, cg, grid, smem, st, pdl);
    if (type == T_Q5_K) return mmq_launch_typed<T_Q5_K>(P, map_w, cg, grid, smem, st, pdl);
    if (type == T_Q6_K) return mmq_launch_typed<T_Q6_K>(P, map_w, cg, grid, smem, st, pdl);
    if (type == T_Q8_0) return mmq_launch_typed<T_Q8_0>(P, map_w, cg, grid, smem, st, pdl);
    return mmq_launch_typed<T_Q5_1>(P, map_w, cg, grid, smem, st, pdl);
}

// d: up to three k-quant matrices with K columns over the activation x, of one type, or of two where one is Q6_K.  One after the other each of them has a
// few tiles to cut into many parts, whose joins and starts take most of the time, and waits for the one in front; together they take a launch.  Not
// supported: where the tiles of all are too many for clusters (74 in halves: K 8192 with 64 + 16 tiles is not), the launches one by one are the faster way by mmq_pick_cut's
// costs, a Q6_K matrix has rows that do not lie at multiples of 16 bytes (K no multiple of 2048), or Q4_K stands beside Q5_K.
// Prompts of models of four layers, one by one / together, widths 2048, 4096 and 5120 with grouped heads: 9 tokens 489 / 404, 749 / 716, 923 / 892; 512 tokens 985 / 802, 1464 / 1280,
// 1788 / 1670.  With as many kv heads as heads at 4096 and 5120, and at 8192, the costs say one by one, and it stays what it was.
// 512 tokens, K 4096, rows 4096 + 1024 + 1024, us: one by one 86, together 42.
cudaError_t launch_mmq_multi(const MmqDesc * d, int n, int64_t K, const float * x, int64_t ldx, int64_t T, void * ws, cudaStream_t st, const MmqPre * pre, bool pdl) {
    if (n < 2 || n > MMQ_MAX_MATS || T <= 0 || K % 256 || K < 256) return cudaErrorNotSupported;
    if (pre && pre->kind != 0 && (!pre->aux || pre->kind < 0 || pre->kind > 2)) return cudaErrorInvalidValue;
    int type = d[0].type, type2 = 0;
    for (int i = 0; i < n; i++) {
        if (!is_kquant(d[i].type) || d[i].N <= 0) return cudaErrorNotSupported;
        if (d[i].type != T_Q6_K) type = d[i].type;
    }
    for (int i = 0; i < n; i++)
        if (d[i].type != type) {
            if (d[i].type != T_Q6_K) return cudaErrorNotSupported;
            type2 = T_Q6_K;
        }
    MmqParams P{};
    MmqMats<true> mats{};
    mats.n = n;
    P.abort_flag = abort_flag();
    P.B = (const uint8_t *) ws;
    P.K = (int) K;
    P.T = (int) T;
    P.BN = mmq_pick_bn((int) T);
    P.ttiles = (int) ((T + P.BN - 1) / P.BN);
    P.nacc = P.ttiles >= 2 ? 2 : 1;
    P.ngrp = (int) (K / 256);
    P.tma = 1;
    const int tgroups = (P.ttiles + P.nacc - 1) / P.nacc, nsm = sm_count();
    const double tokens = (double) std::min<int64_t>(T, 512);
    double apart = 0.0;
    for (int i = 0; i < n; i++) {
        MmqMat & M = mats.mat[i];
        M = MmqMat{(const uint8_t *) d[i].W, d[i].dst, d[i].bias, row_bytes(d[i].type, K), row_bytes(d[i].type, K) * d[i].N, (int) d[i].N, P.rtiles, mmq_group_bytes(d[i].type),
                   mmq_slot_bytes(d[i].type), type2 && d[i].type == type2 ? 1 : 0};
        const int rt = (int) ((d[i].N + MMQ_BM - 1) / MMQ_BM);
        P.rtiles += rt;
        P.slot = std::max(P.slot, M.slot);
        apart += mmq_pick_cut((int64_t) rt * tgroups, P.ngrp, nsm, MMQ_MAX_PARTS, tokens).us;
        if (!mmq_map(mats.map[i], d[i].type, d[i].W, d[i].N, K)) return cudaErrorNotSupported;
    }
    const int64_t tiles = (int64_t) P.rtiles * tgroups;
    if (tiles * P.ngrp > 0x7fffffff) return cudaErrorNotSupported;
    P.total_units = (int) (tiles * P.ngrp);
    const size_t smem = mmq_rings(P, 1);
    if (smem == 0 || (size_t) MMQ_BM * P.BN * 4 > smem - 1024 - MMQ_CTL_BYTES) return cudaErrorNotSupported;
    MmqCut cut = mmq_pick_cut(tiles, P.ngrp, nsm, MMQ_MAX_PARTS, tokens);
    if (cut.parts == 1 && cut.chain == 1 && tiles <= mmq_clusters(2, nsm)) cut.parts = 2;   // halves by a cluster: the same bits
    if (cut.parts < 2 || cut.us >= apart) return cudaErrorNotSupported;
    P.parts = cut.parts;
    const cudaError_t e = mmq_prepare(type, x, ldx, T, K, P.BN, ws, pre, pdl, st);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned) (tiles * cut.parts));
    if (type == T_Q4_K) return type2 ? mmq_launch_typed2<T_Q4_K, 1, true, T_Q6_K>(P, mats, grid, smem, st, pdl) : mmq_launch_typed2<T_Q4_K, 1, true, T_Q4_K>(P, mats, grid, smem, st, pdl);
    if (type == T_Q5_K) return type2 ? mmq_launch_typed2<T_Q5_K, 1, true, T_Q6_K>(P, mats, grid, smem, st, pdl) : mmq_launch_typed2<T_Q5_K, 1, true, T_Q5_K>(P, mats, grid, smem, st, pdl);
    return mmq_launch_typed2<T_Q6_K, 1, true, T_Q6_K>(P, mats, grid, smem, st, pdl);
}

}  // namespace pb
