// prima.cpp_b200/csrc/pdl.h — kernel launches of the layer-list engine that overlap with the kernel in front of them.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace pb {

// Programmatic dependent launch in the layer-list engine.  While it is on (a forward pass of this thread, PdlScope), a kernel launched through
// launch_dep may start when every CTA of the kernel before it on the stream has started, and waits for that kernel's end itself: its launch and
// what it does in front of the wait (weights never depend on the kernel before) lie beside the other's work.  Each such kernel waits in all of
// its threads before it touches anything another kernel writes, so the end of a kernel means the end of all before it; kernels launched the
// plain way (the first of a pass, behind a copy; behind an event of another stream) keep their full dependency.
// What such a kernel reads of an earlier kernel's results it takes by pointers without __restrict__ and by ordinary loads: data that is constant to the
// compiler may be loaded ahead of the wait, wherever the load stands.  Weights and the batch's description (copied in front of the pass) may be.
extern thread_local bool g_pdl;
struct PdlScope {
    bool was;
    explicit PdlScope(bool on) : was(g_pdl) { g_pdl = on; }
    ~PdlScope() { g_pdl = was; }
};
template <typename... P, typename... A>
inline int launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_pdl ? 1 : 0;
    return (int) cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace pb
