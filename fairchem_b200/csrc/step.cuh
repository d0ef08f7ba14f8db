// Pieces shared by the kernels of the whole-model evaluation (edge_step.cuh, node_step.cuh, graph_step.cu) and the host
// code that issues them (model_step.cu).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace fcb200 {

// fcb200_so2_conv_fused for callers in C++; rows_hi, rows_lo: a backward gated list reads the gated rows' planes at its y
// columns in place of y (null: y)
int so2_conv_fused(const void* a_hi, const void* a_lo, int64_t lda, int64_t a_cols, const void* const* w_hi, const void* const* w_lo,
                   const int64_t* w_rows, const int64_t* w_cols, const float* w_scale, const float* const* bias, const int32_t* tiles,
                   int32_t num_tiles, int32_t rot_begin, float* y, int64_t ldy, int64_t y_cols, void* o_hi, void* o_lo, int64_t ldo, int64_t o_cols,
                   const float* a_scale, const float* o_scale, int64_t m, int32_t variant, int32_t* status, void* stream, const __half* rows_hi, const __half* rows_lo, int64_t ld_rows);

namespace step {

constexpr int C = 128;  // channels: sphere, hidden and edge channels of the models this path evaluates

// (a, b) -> packed half pair hi and lo = (v - hi) * 2^11
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn((a - f.x) * 2048.0f, (b - f.y) * 2048.0f);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Largest magnitude of a tensor and the power of two that maps it into (2^5, 2^6], written by the last block of the
// kernel that produces the tensor.  amax and ticket start at zero.
struct Scale {
    uint32_t amax;    // bit pattern of the largest |value|: ordered like the values, so atomicMax applies
    uint32_t ticket;  // blocks that have reported
    float scale;
    float pad;
};

}  // namespace step
}  // namespace fcb200
