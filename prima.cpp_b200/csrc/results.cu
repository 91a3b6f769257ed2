// prima.cpp_b200/csrc/results.cu — page-locked host memory that a model's batch steps hand out for their logits (include/prima_b200.h:
// pb200_result_take / pb200_result_give).  The device writes such rows where the caller reads them; ordinary memory costs a copy through a staging buffer and a
// fault per page of a fresh array: 180 of 582 us of a step that scores 2048 tokens (2 MB), 120 of 640 us of a decode step of eight requests (1 MB).
//
// One pool per model, of a fixed size, taken when the model is finalized.  Blocks may outlive the model: the pool goes with the last of both.  All calls are
// safe from any thread.  The memory is the process's own (registered, not allocated by the driver), in huge pages where the system gives them.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdlib.h>
#include <sys/mman.h>

#include <cstdint>
#include <iterator>
#include <map>
#include <mutex>

#include "../../include/prima_b200.h"
#include "layers.h"

namespace pb {

constexpr size_t RESULT_PAGE = 4096, RESULT_ALIGN = 2u << 20;

struct ResultPool {
    uint8_t * base = nullptr;
    size_t bytes = 0;
    int users = 0;                          // the model and the blocks that are out
    std::map<size_t, size_t> free_, used;   // offset -> bytes
};

namespace {
struct Pools {
    std::mutex lock;
    std::map<uintptr_t, ResultPool *> by_base;
};
Pools & pools() {   // never destroyed: blocks may come back while the process ends
    static Pools * p = new Pools;
    return *p;
}
// the pool, if that was its last user: for unmake, without the lock, which other models' calls share
ResultPool * drop_user(Pools & ps, ResultPool * p) {
    if (--p->users > 0) return nullptr;
    ps.by_base.erase((uintptr_t) p->base);
    return p;
}
void unmake(ResultPool * p) {
    if (!p) return;
    if (cudaHostUnregister(p->base) != cudaSuccess) cudaGetLastError();   // at the process's end the driver may be gone
    free(p->base);
    delete p;
}
}  // namespace

ResultPool * result_pool_create(size_t bytes) {
    bytes = (bytes + RESULT_ALIGN - 1) / RESULT_ALIGN * RESULT_ALIGN;
    void * mem = nullptr;
    if (posix_memalign(&mem, RESULT_ALIGN, bytes) != 0) return nullptr;
    madvise(mem, bytes, MADV_HUGEPAGE);
    if (cudaHostRegister(mem, bytes, cudaHostRegisterPortable) != cudaSuccess) {
        cudaGetLastError();
        free(mem);
        return nullptr;
    }
    ResultPool * p = new ResultPool;
    p->base = (uint8_t *) mem;
    p->bytes = bytes;
    p->users = 1;
    p->free_[0] = bytes;
    Pools & ps = pools();
    std::lock_guard<std::mutex> g(ps.lock);
    ps.by_base[(uintptr_t) mem] = p;
    return p;
}
void result_pool_release(ResultPool * p) {
    if (!p) return;
    Pools & ps = pools();
    {
        std::lock_guard<std::mutex> g(ps.lock);
        p = drop_user(ps, p);
    }
    unmake(p);
}
void * result_take(ResultPool * p, size_t bytes) {
    if (!p || bytes == 0 || bytes > p->bytes) return nullptr;
    bytes = (bytes + RESULT_PAGE - 1) / RESULT_PAGE * RESULT_PAGE;
    std::lock_guard<std::mutex> g(pools().lock);
    for (auto it = p->free_.begin(); it != p->free_.end(); ++it)
        if (it->second >= bytes) {
            const size_t at = it->first, rest = it->second - bytes;
            p->free_.erase(it);
            if (rest) p->free_[at + bytes] = rest;
            p->used[at] = bytes;
            p->users++;
            return p->base + at;
        }
    return nullptr;
}
namespace {
// the driver's page-locked range that holds p (the entry point comes from the driver at run time, nothing links against it)
bool locked_range(const void * p, uintptr_t & start, size_t & size) {
    using Get = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
    static const Get get = [] {
        void * f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return (Get) f;
    }();
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    CUdeviceptr at = 0;
    if (a.type != cudaMemoryTypeHost || !get || get(&at, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, (CUdeviceptr) p) != CUDA_SUCCESS ||
        get(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, (CUdeviceptr) p) != CUDA_SUCCESS)
        return false;
    start = (uintptr_t) at;
    return true;
}
}  // namespace
// One copy takes the whole of [p, p + bytes), so it has to lie in one allocation or registration: two of them side by side, or with ordinary pages between
// them, have page-locked ends as well
bool result_direct(const void * p, size_t bytes) {
    uintptr_t start = 0;
    size_t size = 0;
    if (!p || bytes == 0) return false;
    {
        Pools & ps = pools();
        std::lock_guard<std::mutex> g(ps.lock);
        auto it = ps.by_base.upper_bound((uintptr_t) p);
        if (it != ps.by_base.begin()) {
            --it;
            start = it->first;
            size = it->second->bytes;
        }
    }
    auto holds = [&] { return (uintptr_t) p >= start && bytes <= size && (uintptr_t) p - start <= size - bytes; };
    return holds() || (locked_range(p, start, size) && holds());
}

}  // namespace pb

extern "C" int pb200_result_give(void * block) {
    using namespace pb;
    Pools & ps = pools();
    std::unique_lock<std::mutex> g(ps.lock);
    auto it = ps.by_base.upper_bound((uintptr_t) block);
    if (!block || it == ps.by_base.begin()) return PB200_EINVAL;
    ResultPool * p = (--it)->second;
    auto u = p->used.find((uintptr_t) block - (uintptr_t) p->base);
    if ((uintptr_t) block - (uintptr_t) p->base >= p->bytes || u == p->used.end()) return PB200_EINVAL;
    size_t at = u->first, n = u->second;
    p->used.erase(u);
    auto next = p->free_.lower_bound(at);
    if (next != p->free_.end() && next->first == at + n) { n += next->second; next = p->free_.erase(next); }
    if (next != p->free_.begin()) {
        auto prev = std::prev(next);
        if (prev->first + prev->second == at) { at = prev->first; n += prev->second; p->free_.erase(prev); }
    }
    p->free_[at] = n;
    p = drop_user(ps, p);
    g.unlock();
    unmake(p);
    return 0;
}
