// The network input as the kernels that read it see it: 18 planes of 361 cells
// per position (src/Network.cpp:935-966), fp32, or as bits (18 x 12 words, bit i of
// word w of a plane = cell 32 w + i; every value is 0 or 1).  Bits may lie in
// page-locked host memory: a position is then 864 bytes over the bus, read by the
// kernel that needs them instead of copied and expanded first.
#pragma once
#include "winograd_math.cuh"

namespace lzb {

constexpr int kPlaneWords = 12;

struct InputView {
    const float* f32;              // [n][18][361], or null
    const unsigned int* bits;      // [n][18][12]
    __device__ __forceinline__ float at(int pos, int plane, int s) const {
        if (f32 != nullptr) return f32[(static_cast<size_t>(pos) * kInputPlanes + plane) * kSq + s];
        const unsigned int w = bits[(static_cast<size_t>(pos) * kInputPlanes + plane) * kPlaneWords + (s >> 5)];
        return (w >> (s & 31)) & 1u ? 1.0f : 0.0f;
    }
    __host__ InputView from(int pos) const {
        InputView v = *this;
        if (v.f32 != nullptr) v.f32 += static_cast<size_t>(pos) * kInputPlanes * kSq;
        else v.bits += static_cast<size_t>(pos) * kInputPlanes * kPlaneWords;
        return v;
    }
};

}  // namespace lzb
