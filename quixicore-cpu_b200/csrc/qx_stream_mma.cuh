// Small batches against weights that are streamed once (qx_stream_mma.cu): W8A8, W4A8 and the
// canonical integer layouts.
#pragma once

#include "qx_common.cuh"

namespace qx {

enum StreamSource {
  kStreamBytes,         // [rows][columns] int8, rows on 16 bytes
  kStreamNibbles,       // [rows][columns / 2], lower column in the low nibble, rows on 8 bytes
  kStreamNibblesLoose,  // the same, rows on any byte (int8 activations only)
};

constexpr int kStreamColumns = 64;  // activation rows (digit planes: four or eight per token) at most

constexpr int kStreamW8A8Rows = 32;  // of W8A8

// ---- whole numbers on both sides (one weight scale per row) --------------------------------
// What becomes of a row's exact int32 sums.
enum StreamResult {
  kStreamW8A8,    // (sum - zp[t] * row_sum[o]) * ws[o] * as[t], two rounded multiplies
  kStreamW4A8,    // (sum - 8 * code_sums[t]) * ws[o] * as[t]
  kStreamDigits,  // four or eight digit rows per token: their sums joined, times e[t] * ws[o], bias, activation
};
struct StreamIntArgs {
  StreamSource source;
  StreamResult result;
  const uint8_t* codes;
  const int8_t* x;        // W8A8: [x_rows][columns] int8, rows on 16 bytes; otherwise what the kernels below wrote
  int x_rows;
  int digits;             // digits: rows per token, 4 or 8
  long long rows, columns;
  bool prepared;          // the codes are the library's: they may be read before the kernel in front is done
  const float* ws;        // [rows]
  const float* as;        // [tokens]; eight digits: [tokens][2]
  const int32_t* row_sum; // W8A8 with zero points: [rows], else null
  const int* zp;          // W8A8: [tokens]; W4A8: the code sums [tokens]
  const float* bias;      // digits: [rows] or null
  int activation;
  void* y;                // [tokens][ldy]
  int y_type;
  long long ldy;
  int32_t* acc;           // W8A8: optional [tokens][rows]
};
bool stream_int_serves(const StreamIntArgs& a);
qx_status launch_stream_int(const StreamIntArgs& a, cudaStream_t stream);

// Activations in the order in which the kernel's lanes read them, stream_code_bytes() of them.
// W4A8: codes, scale and sum of the codes per row (quantize_int8, kernels/quantization/quantization_ref.cpp:143-168).
size_t stream_code_bytes(long long x_rows, long long columns);
qx_status launch_stream_codes(const float* x, int8_t* codes, float* scales, int* sums, long long m, long long columns,
                              cudaStream_t stream);
// Digits (columns a multiple of 16). Four rows per token and the envelope: x = e * sum_d 256^d * digit_d to 31 bits of
// the token's largest magnitude. Eight: what that leaves over has an envelope of its own, e[2t] * (the first four +
// e[2t + 1] * the last four), so that a large activation takes no bits from the small ones beside it.
qx_status launch_stream_digits(const void* x, int x_type, int8_t* digits, float* e, long long m, long long columns,
                               int per_token, cudaStream_t stream);

// ---- 16-bit activations, scales along K ------------------------------------------------------
struct StreamScaledArgs {
  StreamSource source;       // bytes or nibbles
  const uint8_t* codes;      // prepared: read before the kernel in front is done
  const float* scales;       // [rows][columns / group]
  const float* zeros;        // nibbles: whole numbers 0 .. 15 beside the scales; null: 8 everywhere
  uint32_t nibble_xor;
  long long rows, columns, group;
  const void* x;             // [m][columns]
  int x_type;                // QX_STORAGE_*
  const int* order;          // optional: packed column -> activation column
  long long m;
  const float* bias;
  int activation;
  void* y;
  int y_type;
  long long ldy;
};
bool stream_scaled_serves(const StreamScaledArgs& a);
// `scratch`: stream_scaled_scratch_bytes() bytes, 16-byte aligned (none: null).
size_t stream_scaled_scratch_bytes(const StreamScaledArgs& a);
qx_status launch_stream_scaled(const StreamScaledArgs& a, void* scratch, cudaStream_t stream);

}  // namespace qx
