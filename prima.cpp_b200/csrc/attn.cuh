// prima.cpp_b200/csrc/attn.cuh — what the attention kernels of the layer-list models share (mixers.cu, attn_decode.cu).
#pragma once
#include "layers.h"
#include "mixers.cuh"

namespace pb {
namespace {

// Cache row of position p: p itself below keep_first, else keep_first + (p - keep_first) mod ring.
__device__ __forceinline__ int cache_row(int p, int keep_first, int ring) { return p < keep_first ? p : keep_first + (p - keep_first) % ring; }
// rows of a slot's cache that hold something for a query at position pi
__device__ __forceinline__ int dec_rows_used(const AttnParams & a, int pi) { return min(a.cache_rows, (a.chunk > 0 ? pi % a.chunk : pi) + 1); }   // a chunk's rows start at row 0 of the ring
// score of the sink of head h
__device__ __forceinline__ float attn_sink(const AttnIO & io, int h) { return io.sink ? io.sink[h] : 0.f; }
// factor on output element d of head h: sigmoid of a gate logit per head, per element, or none
__device__ __forceinline__ float attn_gate(const AttnIO & io, int64_t row, int h, int d, int DV) {
    if (io.gate_mode == 1) return sigmoid_f(io.gate[row * io.ldg + h]);
    if (io.gate_mode == 2) return sigmoid_f(io.gate[row * io.ldg + (int64_t) h * DV + d]);
    return 1.f;
}

}  // namespace
}  // namespace pb
