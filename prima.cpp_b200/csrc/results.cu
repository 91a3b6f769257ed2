// prima.cpp_b200/csrc/results.cu — page-locked host memory that a model's batch steps hand out for their logits (include/prima_b200.h:
// pb200_result_take / pb200_result_give).  The device writes such rows where the caller reads them; ordinary memory costs a copy through a staging buffer and a
// fault per page of a fresh array: 180 of 582 us of a step that scores 2048 tokens (2 MB), 120 of 640 us of a decode step of eight requests (1 MB).
//
// One pool per model, bounded by a fixed size.  It takes its memory slab by slab as blocks are asked for, so that a model whose logits nobody takes from it has none,
// and gives back idle slabs when only that makes room.  Blocks may outlive the model: a slab goes with the last of both.  All calls are safe from any
// thread; slabs are made and unmade outside the lock, which other models' calls share.  The memory is the process's own (registered, not allocated by the driver), in
// huge pages where the system gives them.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdlib.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <iterator>
#include <map>
#include <mutex>
#include <new>
#include <vector>

#include "../../include/prima_b200.h"
#include "layers.h"

namespace pb {

constexpr size_t RESULT_PAGE = 4096, RESULT_ALIGN = 2u << 20;
// A slab holds this many blocks of the size that it is made for, as far as the pool's bound allows: the first step with results waits for it (blocks of 1 MB: 0.4 ms)
constexpr size_t RESULT_SLAB_BLOCKS = 2;

namespace {
struct Slab {
    uint8_t * base = nullptr;
    size_t bytes = 0;
    ResultPool * pool = nullptr;
    std::map<size_t, size_t> free_, used;   // offset -> bytes
};
}  // namespace
struct ResultPool {
    size_t limit = 0, held = 0;             // bytes: the bound, and of the slabs there are or that are being made
    bool closed = false;                    // the model is gone: slabs go as soon as nothing of them is out
    std::vector<Slab *> slabs;
};

namespace {
struct Pools {
    std::mutex lock;
    std::map<uintptr_t, Slab *> by_base;
};
Pools & pools() {   // never destroyed: blocks may come back while the process ends
    static Pools * p = new Pools;
    return *p;
}
// without the lock
bool slab_make(Slab & s, size_t bytes) {
    void * mem = nullptr;
    if (posix_memalign(&mem, RESULT_ALIGN, bytes) != 0) return false;
    madvise(mem, bytes, MADV_HUGEPAGE);
    if (cudaHostRegister(mem, bytes, cudaHostRegisterPortable) != cudaSuccess) {
        cudaGetLastError();
        free(mem);
        return false;
    }
    s.base = (uint8_t *) mem;
    s.bytes = bytes;
    return true;
}
void slabs_unmake(const std::vector<Slab *> & out) {
    for (Slab * s : out) {
        if (cudaHostUnregister(s->base) != cudaSuccess) cudaGetLastError();   // at the process's end the driver may be gone
        free(s->base);
        delete s;
    }
}
// takes the idle slabs out of the pool, for slabs_unmake
void drop_idle(Pools & ps, ResultPool * p, std::vector<Slab *> & out) {
    for (size_t i = 0; i < p->slabs.size();) {
        Slab * s = p->slabs[i];
        if (!s->used.empty()) { i++; continue; }
        out.push_back(s);
        ps.by_base.erase((uintptr_t) s->base);
        p->held -= s->bytes;
        p->slabs.erase(p->slabs.begin() + (ptrdiff_t) i);
    }
}
void * block_of(ResultPool * p, size_t bytes) {
    for (Slab * s : p->slabs)
        for (auto it = s->free_.begin(); it != s->free_.end(); ++it)
            if (it->second >= bytes) {
                const size_t at = it->first, rest = it->second - bytes;
                s->used[at] = bytes;
                if (rest) s->free_[at + bytes] = rest;
                s->free_.erase(at);
                return s->base + at;
            }
    return nullptr;
}
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

ResultPool * result_pool_create(size_t bytes) {
    ResultPool * p = new (std::nothrow) ResultPool;
    if (!p) return nullptr;
    p->limit = (bytes + RESULT_ALIGN - 1) / RESULT_ALIGN * RESULT_ALIGN;
    return p;
}
void result_pool_release(ResultPool * p) {
    if (!p) return;
    std::vector<Slab *> out;
    bool last;
    {
        Pools & ps = pools();
        std::lock_guard<std::mutex> g(ps.lock);
        drop_idle(ps, p, out);
        p->closed = true;
        last = p->slabs.empty();
    }
    slabs_unmake(out);
    if (last) delete p;
}
void * result_take(ResultPool * p, size_t bytes) {
    if (!p || bytes == 0 || bytes > p->limit) return nullptr;
    bytes = (bytes + RESULT_PAGE - 1) / RESULT_PAGE * RESULT_PAGE;
    Pools & ps = pools();
    std::vector<Slab *> out;
    size_t want = (bytes + RESULT_ALIGN - 1) / RESULT_ALIGN * RESULT_ALIGN;
    {
        std::lock_guard<std::mutex> g(ps.lock);
        if (void * b = block_of(p, bytes)) return b;
        size_t idle = 0;
        for (const Slab * s : p->slabs) idle += s->used.empty() ? s->bytes : 0;
        if (p->held - idle + want > p->limit) return nullptr;
        if (p->held + want > p->limit) drop_idle(ps, p, out);   // too small, each of them
        want = std::max(want, std::min((RESULT_SLAB_BLOCKS * bytes + RESULT_ALIGN - 1) / RESULT_ALIGN * RESULT_ALIGN, p->limit - p->held));
        p->held += want;
    }
    slabs_unmake(out);
    Slab * s = new Slab;
    const bool made = slab_make(*s, want);
    std::lock_guard<std::mutex> g(ps.lock);
    if (!made) {
        p->held -= want;
        delete s;
        return nullptr;
    }
    s->pool = p;
    s->used[0] = bytes;
    if (want > bytes) s->free_[bytes] = want - bytes;
    p->slabs.push_back(s);
    ps.by_base[(uintptr_t) s->base] = s;
    return s->base;
}
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

extern "C" int pb200_result_give(void * block) try {
    using namespace pb;
    Pools & ps = pools();
    std::vector<Slab *> out;
    ResultPool * last = nullptr;
    {
        std::lock_guard<std::mutex> g(ps.lock);
        auto it = ps.by_base.upper_bound((uintptr_t) block);
        if (!block || it == ps.by_base.begin()) return PB200_EINVAL;
        Slab * s = (--it)->second;
        auto u = s->used.find((uintptr_t) block - (uintptr_t) s->base);
        if ((uintptr_t) block - (uintptr_t) s->base >= s->bytes || u == s->used.end()) return PB200_EINVAL;
        size_t at = u->first, n = u->second;
        s->used.erase(u);
        auto next = s->free_.lower_bound(at);
        if (next != s->free_.end() && next->first == at + n) { n += next->second; next = s->free_.erase(next); }
        if (next != s->free_.begin()) {
            auto prev = std::prev(next);
            if (prev->first + prev->second == at) { at = prev->first; n += prev->second; s->free_.erase(prev); }
        }
        s->free_[at] = n;
        ResultPool * p = s->pool;
        if (p->closed) {
            drop_idle(ps, p, out);
            if (p->slabs.empty()) last = p;
        }
    }
    slabs_unmake(out);
    delete last;
    return 0;
} catch (...) {   // no memory for the bookkeeping
    return PB200_ENOMEM;
}
