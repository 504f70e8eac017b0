// Batched projections whose weight scales change along K, on the tensor cores
// (qx_scaled_gemm.cu): canonical int4 / uint4 / int8 tensors and prepared q8_0 panels.
#pragma once

#include "qx_common.cuh"

namespace qx {

enum ScaledGemmSource {
  kScaledNibbles,  // [rows][columns / 2] bytes, lower column in the low nibble, f32 scales
  kScaledBytes,    // [rows][columns] int8, f32 scales
  kScaledPanelQ8,  // prepared q8_0 panel (qx_weights.cuh), fp16 scales inside
  kScaledNibblesLoose  // as kScaledNibbles, rows that start on any byte
};

struct ScaledGemmArgs {
  ScaledGemmSource source;
  const uint8_t* codes;      // device: codes or panel
  const float* scales;       // [rows][columns / group] below 2^111 (not for the panel)
  const float* zeros;        // nibbles: zero point beside every scale, whole numbers 0 .. 15;
                             // null: 8 everywhere
  uint32_t nibble_xor;       // 0x88888888 for two's complement nibbles, else 0
  long long rows, columns;
  long long group;           // columns per scale: a multiple of 32, or `columns` (one per row)
  const void* x;             // [m][columns]
  int x_type;                // QX_STORAGE_*
  const int* order;          // optional: packed column -> activation column
  long long m;
  const float* bias;         // [rows] or null
  int activation;
  const float* token_scales; // [m] or null. Given: x holds whole numbers and the result is
                             // (sum * scales[row]) * token_scales[token], two rounded multiplies
                             // of an exact sum (one scale per row, f16 activations)
  long long x_stride;        // elements between activation rows; 0: columns
  bool whole_tiles;          // no pieces of tiles (they need scratch)
  void* y;                   // [m][ldy]
  int y_type;
  long long ldy;
};

// Whether the sizes and pointers are ones that the kernel takes (not whether it is the better
// choice: that is the caller's rule).
bool scaled_gemm_serves(const ScaledGemmArgs& a);
// Scratch behind the workspace's counters for launch_scaled_gemm(): enough for `a` and for every
// call of fewer tokens, of any type and alignment, on the same tensor, so that a workspace which
// has served the largest batch does not grow any more (it could not under stream capture).
size_t scaled_gemm_scratch_bytes(const ScaledGemmArgs& a, int sm_count);
// Bytes of counters that a launch of at most `ctas` CTAs uses: a CTA holds the first piece of at
// most two tiles, and every epilogue warp counts for itself.
constexpr int kScaledEpilogueWarps = 16;  // of the shape that has most of them
constexpr size_t scaled_gemm_counter_bytes(int ctas) {
  return 2 * static_cast<size_t>(ctas) * kScaledEpilogueWarps * sizeof(int);
}
// `scratch`: scaled_gemm_scratch_bytes() bytes, 256-byte aligned; `counters`: `counter_bytes` of
// zeroed counters (fewer than the launch needs: QX_STATUS_DEVICE_ERROR), left zeroed.
qx_status launch_scaled_gemm(const ScaledGemmArgs& a, void* scratch, int* counters, size_t counter_bytes,
                             int sm_count, int* error, cudaStream_t stream);

// Storage types and activations of a projection's epilogue (qx_canonical.cu), shared.
__device__ __forceinline__ uint16_t storage_bf16_bits(float value) {
  // float_to_bf16 of the reference (kernels/utils/float_storage_ref.cpp:184-193): round to
  // nearest even on the bit pattern; a NaN keeps its upper payload with the quiet bit set.
  const uint32_t bits = __float_as_uint(value);
  if ((bits & 0x7f800000u) == 0x7f800000u && (bits & 0x007fffffu) != 0) {
    return static_cast<uint16_t>((bits >> 16) | 0x0040u);
  }
  return static_cast<uint16_t>((bits + 0x7fffu + ((bits >> 16) & 1u)) >> 16);
}
// projection_activation, qgemm_canonical.cpp:361-379
__device__ __forceinline__ float projection_activation(float v, int activation) {
  switch (activation) {
    case QX_ACTIVATION_GELU_ERF:
      return 0.5f * v * (1.0f + erff(v * 0.7071067811865475f));
    case QX_ACTIVATION_GELU_TANH:
      return 0.5f * v * (1.0f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
    case QX_ACTIVATION_SILU:
      return v / (1.0f + expf(-v));
    case QX_ACTIVATION_RELU2:
      return v > 0.0f ? v * v : 0.0f;
    default:
      return v;
  }
}

}  // namespace qx
