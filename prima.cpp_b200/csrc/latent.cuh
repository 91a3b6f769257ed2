// prima.cpp_b200/csrc/latent.cuh — what the kernels of attention over a latent share (latent.cu, latent_decode.cu).
#pragma once
#include <math.h>

#include "layers.h"
#include "mixers.cuh"

namespace pb {
namespace {

// entries of pair i
__device__ __forceinline__ void pair_at(const LatentParams & p, int i, int & ia, int & ib) {
    if (p.rot_layout == ROT_INTERLEAVED) { ia = 2 * i; ib = 2 * i + 1; }
    else { ia = i; ib = i + p.rot_dims / 2; }
}
// rotates the pair (u, v) by the angle pos * freq; cos and sin carry the factor mag
__device__ __forceinline__ void turn(float u, float v, int pos, float f, float mag, float & ou, float & ov) {
    const float ang = (float) pos * f;
    const float c = cosf(ang) * mag, s = sinf(ang) * mag;
    ou = u * c - v * s;
    ov = v * c + u * s;
}

// factor on output element (head h, entry dv): sigmoid of the head's gate logit, of the element's, or none
__device__ __forceinline__ float latent_gate(const LatentParams & p, const float * gate, int64_t at, int h, int dv) {
    return gate ? sigmoid_f(gate[at + (p.gate_mode == 1 ? h : h * p.vdim + dv)]) : 1.f;
}

}  // namespace
}  // namespace pb
