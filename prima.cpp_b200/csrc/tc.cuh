// prima.cpp_b200/csrc/tc.cuh — what the kernels on the 5th-generation tensor cores share: tcgen05 instructions, shared-memory descriptors, tiled TMA
// loads and the tensor maps they need.
//
// A role that issues asynchronous instructions runs as a whole warp through its loop and elects a lane for each group of instructions:
// addresses and descriptors stay in uniform registers then.  A loop inside `if (lane == 0)` moves every operand there again: 54 clocks an MMA
// were measured, 4 of them, a commit and a wait being 350 clocks of a step whose MMAs take 256 (128 x 128 x 64).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "common.cuh"

namespace pb {
namespace {

__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n"
        ".reg .pred q;\n"
        "elect.sync _|q, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, q;\n"
        "}\n"
        : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int) (threadIdx.x >> 5), 0); }

// operand in shared memory, K-major, SWIZZLE_128B: rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
    uint64_t d = (uint64_t) ((saddr >> 4) & 0x3FFF);
    d |= (uint64_t) 1 << 16;
    d |= (uint64_t) (1024 >> 4) << 32;
    d |= (uint64_t) 1 << 46;
    d |= (uint64_t) 2 << 61;
    return d;
}
template <int CG>
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    if constexpr (CG == 1)
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "setp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
            "}\n" ::"r"(tmem_d),
            "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "setp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
            "}\n" ::"r"(tmem_d),
            "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
            : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t * bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// completion of all prior MMAs of the pair -> the barrier at this offset in both CTAs
__device__ __forceinline__ void mma_commit_pair(uint64_t * bar) {
    const uint16_t mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(mask)
                 : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t saddr, uint32_t rank) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(saddr), "r"(rank));
    return ra;
}
// a number into the same place of another CTA's shared memory
__device__ __forceinline__ void send(float v, const float * at, int cta) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr(smem_u32(at), (uint32_t) cta)), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap * m) { asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory"); }
// a box at (x, y, z); bar: shared-memory address in the cluster's window (CG 2: either CTA of the pair)
template <int CG>
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap * m, int x, int y, int z, uint32_t bar) {
    if constexpr (CG == 1)
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(m), "r"(x),
                     "r"(y), "r"(z), "r"(bar)
                     : "memory");
    else
        asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(m),
                     "r"(x), "r"(y), "r"(z), "r"(bar)
                     : "memory");
}
// the warp's 32 lanes x 16 columns of an accumulator, waited for
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
          "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {   // A in tensor memory
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// operand in shared memory, N contiguous (values [key][dim]), SWIZZLE_128B: rows of 64 entries, 8-key groups 1024 bytes apart, blocks of 64 entries `block` bytes apart
__device__ __forceinline__ uint64_t desc_sw128_mn(uint32_t saddr, uint32_t block) {
    uint64_t d = (uint64_t) ((saddr >> 4) & 0x3FFF);
    d |= (uint64_t) (block >> 4) << 16;
    d |= (uint64_t) (1024 >> 4) << 32;
    d |= (uint64_t) 1 << 46;
    d |= (uint64_t) 2 << 61;
    return d;
}
#define TMEM_LD32(addr, v)                                                                                                                              \
    asm volatile(                                                                                                                                       \
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "   \
        "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"                                                                                     \
        : "=r"((v)[0]), "=r"((v)[1]), "=r"((v)[2]), "=r"((v)[3]), "=r"((v)[4]), "=r"((v)[5]), "=r"((v)[6]), "=r"((v)[7]), "=r"((v)[8]), "=r"((v)[9]),     \
          "=r"((v)[10]), "=r"((v)[11]), "=r"((v)[12]), "=r"((v)[13]), "=r"((v)[14]), "=r"((v)[15]), "=r"((v)[16]), "=r"((v)[17]), "=r"((v)[18]),          \
          "=r"((v)[19]), "=r"((v)[20]), "=r"((v)[21]), "=r"((v)[22]), "=r"((v)[23]), "=r"((v)[24]), "=r"((v)[25]), "=r"((v)[26]), "=r"((v)[27]),          \
          "=r"((v)[28]), "=r"((v)[29]), "=r"((v)[30]), "=r"((v)[31])                                                                                    \
        : "r"(addr)                                                                                                                                     \
        : "memory")
#define TMEM_ST16(addr, v)                                                                                                                              \
    asm volatile(                                                                                                                                       \
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr), "r"((v)[0]), \
        "r"((v)[1]), "r"((v)[2]), "r"((v)[3]), "r"((v)[4]), "r"((v)[5]), "r"((v)[6]), "r"((v)[7]), "r"((v)[8]), "r"((v)[9]), "r"((v)[10]), "r"((v)[11]),  \
        "r"((v)[12]), "r"((v)[13]), "r"((v)[14]), "r"((v)[15])                                                                                          \
        : "memory")
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ---- host: tensor maps (the encoder comes from the driver at run time, nothing links against it) ----
using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                 CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void * p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return (EncodeTiled) p;
    }();
    return fn;
}
// planes x rows x cols of a 16-bit type (rows ld elements apart, planes `plane`), boxes of 64 columns x box_rows in the swizzle-128B image; what lies
// outside reads zeros
inline int make_map(CUtensorMap & m, CUtensorMapDataType type, const void * base, int64_t cols, int64_t rows, int64_t planes, int64_t ld, int64_t plane, int box_rows) {
    const EncodeTiled fn = encode_tiled();
    if (!fn) return (int) cudaErrorNotSupported;
    const cuuint64_t dims[3] = {(cuuint64_t) cols, (cuuint64_t) rows, (cuuint64_t) planes};
    const cuuint64_t strides[2] = {(cuuint64_t) ld * 2, (cuuint64_t) (planes > 1 ? plane : rows * ld) * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t) box_rows, 1}, one[3] = {1, 1, 1};
    const CUresult r = fn(&m, type, 3, (void *) base, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int) cudaErrorInvalidValue;
}

}  // namespace
}  // namespace pb
