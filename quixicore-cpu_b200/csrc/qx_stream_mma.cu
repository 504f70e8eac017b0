// Small batches (up to 64 activation rows) against weights that are streamed once:
//   int8_gemm / qgemm_w8a8   kernels/quantization/int8_gemm_ref.cpp:9-32           (exact)
//   lowbit_gemm_w8a8         kernels/quantization/lowbit_w8a8_ref.cpp:7-32         (exact)
//   qgemm_prepacked_epilogue_storage on the canonical integer layouts
//                            kernels/quantization/qgemm_canonical.cpp:4460-4648
//
// What bounds such a call is how fast the codes come from memory, and for matrices of a few MB
// the fixed costs around that. A pipeline of specialised warps over 128-row tiles (qx_scaled_gemm.cu,
// qx_int8_gemm_tc.cu) has few CTAs here and 8 us of start and end. So: no shared memory and no
// barriers on the way of the weights. A warp owns 16 or 32 weight rows and one contiguous part of
// K (eight warps of a CTA share the rows); its lanes load codes straight into registers, two
// or four steps ahead, in the places where the warp-level MMA wants them as its A operand: lane (g, t)
// holds rows g and g + 8 and a quarter of a step's columns, in one piece. Which columns an MMA slot
// stands for is free as long as both operands agree: the B operand is read through L1 with 16-byte loads,
// from the activations' rows as they are (W8A8, up to eight 16-bit tokens), or where a kernel in front
// writes them anyway, or for more tokens, from the order in which the lanes read them (plain rows cost a
// load eight lines). The parts of K meet in shared memory at the end, in exact integers or in 64 bits.
//
// Measured (us, before | here, codes from memory): W4A8 16 rows 4096 x 4096 22.6 | 8.2; W8A8 4 rows 1024 x 1408 6.0 | 3.0; int8
// 1 token 14336 x 4096 17.3 | 16.1 (3.7 TB/s); uint4 16 tokens 14336 x 4096 32.2 | 23.5. 16-bit activations are bound
// by the latency of loads at four warps per scheduler (more than half of the cycles between two instructions of a
// warp), which the registers of 32 rows x 16 tokens leave no room to ask for earlier.
//
// tcgen05 would need both operands in shared memory and a TMEM round trip per scale group; at
// these batch sizes the tensor work is a few percent of what either path could do.
//
// Whole numbers (launch_stream_int): m16n8k32 s8 x s8 or u8 x s8 (nibbles as they are, the -8 of
// the format through the activations' sums), int32 sums over the whole row. A canonical int8 tensor's
// activations enter as four digit rows per token (31-bit fixed point under the token's envelope,
// as canonical_row_digits_kernel has it), joined in 64-bit integers. Up to four tokens have eight: the digit kernel for
// such batches gives every 16 columns an envelope of their own, and with one for the whole token an activation
// 2^20 times the others would leave them ten bits (5.6e-4 of a result that does not see the large one). The second four
// rows are the remainders under the remainders' envelope; they fill MMA columns that would be padding for one token.
//
// 16-bit activations (launch_stream_scaled): the arithmetic of qx_scaled_gemm.cu: whole numbers of
// at most eight bits times f16 or bf16, sums of at most 128 columns (64 with three planes, 32 of
// bytes with f16) by the tensor core, each scaled by an f32 multiply-add.

#include "qx_scaled_gemm.cuh"
#include "qx_stream_mma.cuh"
#include "qx_tile_pipe.cuh"

namespace qx {
namespace {

using tile::wait_for_kernel_in_front;

constexpr int kWarps = 8;
constexpr int kThreads = 32 * kWarps;

__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }

// D += A * B, 16 x 8 outputs
template <bool UNSIGNED_A>
__device__ __forceinline__ void mma_i8(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b0, uint32_t b1) {
  if (UNSIGNED_A) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}
template <bool BF16>
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
  if (BF16) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}

// Codes pass through once: they leave L1 to the activations.
__device__ __forceinline__ void load_words(const uint8_t* src, uint32_t (&w)[1]) {
  asm volatile("ld.global.b32 %0, [%1];" : "=r"(w[0]) : "l"(src));  // (half a sector per row: the other half follows)
}
__device__ __forceinline__ void load_words(const uint8_t* src, uint32_t (&w)[2]) {
  asm volatile("ld.global.L1::no_allocate.v2.b32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "l"(src));
}
__device__ __forceinline__ void load_words(const uint8_t* src, uint32_t (&w)[4]) {
  asm volatile("ld.global.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
               : "l"(src));
}
// Eight bytes on an 8-byte boundary of which some may lie outside [begin, end): those read as zero.
__device__ __forceinline__ void load_guarded(const uint8_t* src, const uint8_t* begin, const uint8_t* end,
                                             uint32_t& w0, uint32_t& w1) {
  if (src >= begin && src + 8 <= end) {
    asm volatile("ld.global.v2.b32 {%0, %1}, [%2];" : "=r"(w0), "=r"(w1) : "l"(src));
    return;
  }
  w0 = w1 = 0u;
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    if (src + i >= begin && src + i < end) {
      const uint32_t v = static_cast<uint32_t>(src[i]) << (8 * (i & 3));
      if (i < 4) w0 |= v; else w1 |= v;
    }
  }
}
__device__ __forceinline__ uint4 load_activations(const uint8_t* src) {
  uint4 v;
  asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(src));
  return v;
}

// Calls a CTA's rows of codes into L2. Before the wait for the kernel in front this reads nothing
// on the program's behalf: should that kernel write these bytes, the lines in L2 change with them.
// Matrices of up to 32 MB as a whole. Of larger ones the requests of all CTAs stand in the way of the loads: the first 24 MB
// of whole numbers, whose first CTAs wait for the kernel in front anyway, and nothing with scales along K. Measured (us, none |
// 24 MB | all; graph replay, codes from memory): int8 one token 4096 x 4096 7.3 | 6.9 | 6.9, 14336 x 4096 16.8 | 16.1 | 17.5,
// 28672 x 8192 54 | 52 | 67, 8192 x 16384 33.5 | 30.8 | 35.1, W8A8 1024 x 28672 34.3 | 36.5 | 35.4;  uint4 five tokens
// 4096 x 14336 18.8 | 20.7 | 19.9, 16 tokens 14336 x 4096 23.2 | 23.3 | 23.5, 28672 x 8192 78 | 79 | 88. Three matrices in
// turn, partly in L2: W8A8 1024 x 28672 33.1 | 34.5 | 28.0, int8 14336 x 4096 17.1 | 16.2 | 15.5, uint4 five tokens 18.5 |
// 18.4 | 17.4.
// (`rows` 0: an empty range and not a branch around the loop, behind which the loads of 16 uint4 tokens with groups of 32 on
// 11008 x 4096 took 45 us, not 38.)
constexpr long long kPrefetchWhole = 1LL << 25, kPrefetchFirst = 24LL << 20;
__device__ __forceinline__ void prefetch_rows(const uint8_t* codes, long long row_bytes, long long row0, int rows,
                                              long long total_rows) {
  const long long last = row0 + rows < total_rows ? row0 + rows : total_rows;
  const uintptr_t begin = (reinterpret_cast<uintptr_t>(codes + row0 * row_bytes) + 15) & ~uintptr_t(15);
  const uintptr_t end = reinterpret_cast<uintptr_t>(codes + last * row_bytes) & ~uintptr_t(15);
  constexpr uintptr_t kPiece = 16 * 1024;
  for (uintptr_t at = begin + threadIdx.x * kPiece; at < end; at += kThreads * kPiece) {
    const uint32_t size = static_cast<uint32_t>(end - at < kPiece ? end - at : kPiece);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at), "r"(size));
  }
}

__device__ __forceinline__ void store_output(void* y, int type, long long index, float value) {
  if (type == QX_STORAGE_F32) {
    static_cast<float*>(y)[index] = value;
  } else {
    static_cast<uint16_t*>(y)[index] =
        type == QX_STORAGE_F16 ? __half_as_ushort(__float2half_rn(value)) : storage_bf16_bits(value);
  }
}

// ---- whole numbers ---------------------------------------------------------------------------
struct IntParams {
  const uint8_t* codes;
  const uint8_t* codes_end;
  const uint8_t* x;
  const float* ws;
  const float* as;
  const int32_t* row_sum;
  const int* zp;
  const float* bias;
  void* y;
  int32_t* acc;
  long long row_bytes, x_stride, ldy;
  int rows, columns, x_rows, steps;
  int prefetch_rows, activation, y_type, prepared, digits;
};

// A step is 64 columns: 16 per lane of a quad (16 bytes of int8, 8 bytes of nibbles).
template <StreamSource SRC, bool FRAGMENTS, int NT, int MR, int AHEAD, int CTAS>
__global__ void __launch_bounds__(kThreads, CTAS) stream_int_kernel(const IntParams p) {
  constexpr bool kLoose = SRC == kStreamNibblesLoose;
  constexpr bool kNibbles = SRC != kStreamBytes;
  constexpr int kWords = SRC == kStreamNibbles ? 2 : 4;  // loose: the 16 bytes around a row's 8
  constexpr int kR = 16 * MR;
  // (what becomes of the sums goes with the source: digits lie in the lanes' order beside bytes, W8A8 activations as they are)
  constexpr bool kDigits = SRC == kStreamBytes && FRAGMENTS;
  __shared__ int red[kWarps][kR][9];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int row0 = blockIdx.x * kR;
  launch_dependents();
  prefetch_rows(p.codes, p.row_bytes, row0, row0 < p.prefetch_rows ? kR : 0, p.rows);

  // (offsets from the CTA's first row: a pointer per row would be two registers)
  const uint8_t* codes = p.codes + row0 * p.row_bytes + t * (kNibbles ? 8 : 16);
  const int slack = kLoose ? static_cast<int>(reinterpret_cast<uintptr_t>(codes) & 7u) : 0;
  codes -= slack;
  uint32_t code_at[MR][2], shift[MR][2];
#pragma unroll
  for (int i = 0; i < MR; ++i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // (a row past the last one repeats it: its sums are not stored)
      const int row = min(16 * i + 8 * h + g, p.rows - 1 - row0);
      code_at[i][h] = static_cast<uint32_t>(row) * static_cast<uint32_t>(p.row_bytes) + slack;
      if (kLoose) {
        shift[i][h] = code_at[i][h] & 7u;
        code_at[i][h] &= ~7u;
      }
    }
  }
  const int s0 = p.steps * warp / kWarps, s1 = p.steps * (warp + 1) / kWarps;
  uint32_t ring[AHEAD][MR][2][kWords];
  auto fetch = [&](uint32_t (&into)[MR][2][kWords], int step) {
    const int column = step * 64 + t * 16;
#pragma unroll
    for (int i = 0; i < MR; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint8_t* at = codes + (code_at[i][h] + step * (kNibbles ? 32 : 64));
        if (column < p.columns) {
          if constexpr (kLoose) {
            load_guarded(at, p.codes, p.codes_end, into[i][h][0], into[i][h][1]);
            load_guarded(at + 8, p.codes, p.codes_end, into[i][h][2], into[i][h][3]);
          } else {
            load_words(at, into[i][h]);
          }
        } else {
#pragma unroll
          for (int q = 0; q < kWords; ++q) into[i][h][q] = 0u;
        }
      }
    }
  };
  if (!p.prepared) wait_for_kernel_in_front();  // the codes may be that kernel's output
#pragma unroll
  for (int d = 0; d < AHEAD; ++d) {
    if (s0 + d < s1) fetch(ring[d], s0 + d);
  }
  if (p.prepared) wait_for_kernel_in_front();
  const uint8_t* x_at[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    // (likewise a column past the last one)
    x_at[n] = FRAGMENTS ? p.x + (n * 32 + lane) * 16 : p.x + min(8 * n + g, p.x_rows - 1) * p.x_stride + t * 16;
  }
  uint32_t sum[MR][NT][4];
#pragma unroll
  for (int i = 0; i < MR; ++i) {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[i][n][c] = 0u;
    }
  }
  // (the activations of a step are asked for before the products of the one in front of it)
  constexpr bool kEarly = NT <= 4;
  uint4 ahead[NT];
  auto fetch_x = [&](int step) {
    const bool inside = step < s1 && (FRAGMENTS || step * 64 + t * 16 < p.columns);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      ahead[n] = make_uint4(0u, 0u, 0u, 0u);
      if (inside) ahead[n] = load_activations(x_at[n] + step * (FRAGMENTS ? NT * 512 : 64));
    }
  };
  if (kEarly) fetch_x(s0);
  for (int s = s0; s < s1; s += AHEAD) {
#pragma unroll
    for (int d = 0; d < AHEAD; ++d) {
      const int step = s + d;
      if (step < s1) {
        uint4 b[NT];
        if (!kEarly) fetch_x(step);
#pragma unroll
        for (int n = 0; n < NT; ++n) b[n] = ahead[n];
        if (kEarly) fetch_x(step + 1);
        uint32_t a[MR][2][4];  // [row half][two words per MMA]
#pragma unroll
        for (int i = 0; i < MR; ++i) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t (&w)[kWords] = ring[d][i][h];
            if constexpr (SRC == kStreamBytes) {
#pragma unroll
              for (int q = 0; q < 4; ++q) a[i][h][q] = w[q];
            } else {
              uint32_t v[2] = {w[0], w[1]};
              if constexpr (kLoose) {
                const bool upper = (shift[i][h] & 4u) != 0;
                const uint32_t bits = (shift[i][h] & 3u) * 8;
                const uint32_t v0 = upper ? w[1] : w[0], v1 = upper ? w[2] : w[1], v2 = upper ? w[3] : w[2];
                v[0] = __funnelshift_r(v0, v1, bits);
                v[1] = __funnelshift_r(v1, v2, bits);
              }
#pragma unroll
              for (int q = 0; q < 2; ++q) {  // even columns, odd columns
                a[i][h][2 * q] = v[q] & 0x0F0F0F0Fu;
                a[i][h][2 * q + 1] = (v[q] >> 4) & 0x0F0F0F0Fu;
              }
            }
          }
        }
        if (step + AHEAD < s1) fetch(ring[d], step + AHEAD);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
#pragma unroll
          for (int i = 0; i < MR; ++i) {
            mma_i8<kNibbles>(sum[i][n], a[i][0][0], a[i][1][0], a[i][0][1], a[i][1][1], b[n].x, b[n].y);
            mma_i8<kNibbles>(sum[i][n], a[i][0][2], a[i][1][2], a[i][0][3], a[i][1][3], b[n].z, b[n].w);
          }
        }
      }
    }
  }
  // eight columns at a time: the warps' parts of K are added, exactly
  const int r = threadIdx.x % kR;
  const int row = row0 + r;
  // Digits per token: one token of eight columns, or two. One and two tokens have eight, nine and more four.
  const bool eight = NT <= 2 || (NT == 4 && p.digits == 8);
  const int digit_at = threadIdx.x / kR;
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int digit_token = eight ? n : 2 * n + digit_at;
    const bool digit_mine = kDigits && digit_at < (eight ? 1 : 2) && row < p.rows &&
                            digit_token * (eight ? 8 : 4) < p.x_rows;
    float digit_e = 0.0f, digit_rest = 0.0f, digit_ws = 0.0f;
    if (digit_mine) {  // (asked for before the sums meet)
      digit_e = p.as[eight ? 2 * digit_token : digit_token];
      if (eight) digit_rest = p.as[2 * digit_token + 1];
      digit_ws = __ldg(p.ws + row);
    }
    if (n > 0) __syncthreads();
#pragma unroll
    for (int i = 0; i < MR; ++i) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        red[warp][16 * i + 8 * (c >> 1) + g][2 * t + (c & 1)] = static_cast<int>(sum[i][n][c]);
      }
    }
    __syncthreads();
    if constexpr (kDigits) {
      if (digit_mine) {
        auto joined = [&](int first) {  // four digits
          long long total = 0;
#pragma unroll
          for (int d = 3; d >= 0; --d) {
            int part = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) part += red[w][r][first + d];
            total = total * 256 + part;
          }
          return static_cast<double>(total);
        };
        double total = joined(eight ? 0 : 4 * digit_at);
        if (eight) total += joined(4) * static_cast<double>(digit_rest);
        // (a token that holds a value that is not finite has a NaN for its envelope)
        float out = static_cast<float>(total * (static_cast<double>(digit_e) * static_cast<double>(digit_ws)));
        if (p.bias != nullptr) out += __ldg(p.bias + row);
        if (p.activation != QX_ACTIVATION_NONE) out = projection_activation(out, p.activation);
        store_output(p.y, p.y_type, digit_token * p.ldy + row, out);
      }
    } else {
      const int token = 8 * n + threadIdx.x / kR;
      if (threadIdx.x < 8 * kR && row < p.rows && token < p.x_rows) {
        int total = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) total += red[w][r][token & 7];
        float value;
        if constexpr (kNibbles) {
          value = static_cast<float>(total - 8 * p.zp[token]);
        } else {
          long long dot = total;
          if (p.row_sum != nullptr) dot -= static_cast<long long>(p.zp[token]) * p.row_sum[row];
          value = p.row_sum != nullptr ? __ll2float_rn(dot) : __int2float_rn(total);
          if (p.acc != nullptr) p.acc[static_cast<long long>(token) * p.rows + row] = static_cast<int32_t>(dot);
        }
        static_cast<float*>(p.y)[token * p.ldy + row] = __fmul_rn(__fmul_rn(value, p.ws[row]), p.as[token]);
      }
    }
  }
}

// ---- 16-bit activations, scales along K --------------------------------------------------------
struct ScaledParams {
  const uint8_t* codes;
  const uint8_t* x;
  const float* scales;
  const float* zeros;
  const float* bias;
  void* y;
  long long row_bytes, x_stride, ldy;
  uint32_t nibble_xor;
  int rows, columns, m, steps, group, groups, flush_steps;
  int prefetch_rows, activation, y_type;
};

// A step is 64 columns, or 32 where sums of 32 leave the tensor core: a quarter per lane of a quad.
template <StreamSource SRC, bool FRAGMENTS, bool BF16, int PLANES, int STEP, int NT, int MR, int AHEAD, int CTAS>
__global__ void __launch_bounds__(kThreads, CTAS) stream_scaled_kernel(const ScaledParams p) {
  constexpr bool kNibbles = SRC == kStreamNibbles;
  constexpr int kColumns = STEP / 4;                       // of a lane
  constexpr int kBytes = kNibbles ? kColumns / 2 : kColumns;
  constexpr int kWords = kBytes / 4;
  constexpr int kFrags = kColumns / 8;
  // activations asked for one step ahead, where that spills nothing (two tiles of rows, uint4, 16 tokens on 14336 x 4096:
  // 25.4 us with it, 22.8 without; one tile of rows, 4096 x 4096: 7.8 against 10.0)
  constexpr bool kEarly = PLANES == 1 && MR == 1 && NT * kFrags <= 4;
  constexpr int kR = 16 * MR;
  constexpr int kPitch = 8 * NT + 1;
  __shared__ float red[kWarps][kR][kPitch];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int row0 = blockIdx.x * kR;
  launch_dependents();
  prefetch_rows(p.codes, p.row_bytes, row0, row0 < p.prefetch_rows ? kR : 0, p.rows);

  // (offsets from the CTA's first row: a pointer per row would be two registers)
  const uint8_t* codes = p.codes + row0 * p.row_bytes + t * kBytes;
  const float* scales = p.scales + static_cast<long long>(row0) * p.groups;
  const float* zeros = kNibbles && p.zeros != nullptr ? p.zeros + static_cast<long long>(row0) * p.groups : nullptr;
  uint32_t code_at[MR][2], scale_at[MR][2];
#pragma unroll
  for (int i = 0; i < MR; ++i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // (a row past the last one repeats it: its sums are not stored)
      const int row = min(16 * i + 8 * h + g, p.rows - 1 - row0);
      code_at[i][h] = static_cast<uint32_t>(row) * static_cast<uint32_t>(p.row_bytes);
      scale_at[i][h] = static_cast<uint32_t>(row) * static_cast<uint32_t>(p.groups);
    }
  }
  const int s0 = p.steps * warp / kWarps, s1 = p.steps * (warp + 1) / kWarps;
  uint32_t ring[AHEAD][MR][2][kWords];
  auto fetch = [&](uint32_t (&into)[MR][2][kWords], int step) {
    const bool inside = step * STEP + t * kColumns < p.columns;
#pragma unroll
    for (int i = 0; i < MR; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (inside) {
          load_words(codes + (code_at[i][h] + step * (4 * kBytes)), into[i][h]);
        } else {
#pragma unroll
          for (int q = 0; q < kWords; ++q) into[i][h][q] = 0u;
        }
      }
    }
  };
#pragma unroll
  for (int d = 0; d < AHEAD; ++d) {
    if (s0 + d < s1) fetch(ring[d], s0 + d);
  }
  // scale and zero point of the group at hand, and of the next one
  int group = s0 < s1 ? s0 * STEP / p.group : 0;
  int boundary = (group + 1) * p.group;
  float scale[MR][2], next_scale[MR][2], next_zero[MR][2];
  uint32_t base_z[MR][2];
  auto fetch_group = [&](int which) {
#pragma unroll
    for (int i = 0; i < MR; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        next_scale[i][h] = __ldg(scales + (scale_at[i][h] + which));
        next_zero[i][h] = zeros != nullptr ? __ldg(zeros + (scale_at[i][h] + which)) : 8.0f;
      }
    }
  };
  auto take_group = [&]() {
#pragma unroll
    for (int i = 0; i < MR; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        scale[i][h] = BF16 ? next_scale[i][h] * tile::kBf16Unscale : next_scale[i][h];
        if (kNibbles) base_z[i][h] = tile::zero_word<BF16>(next_zero[i][h]);
      }
    }
  };
  fetch_group(group);
  take_group();
  fetch_group(min(group + 1, p.groups - 1));
  const uint8_t* x_at[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    // (likewise a token past the last one)
    x_at[n] = FRAGMENTS ? p.x + (n * 32 + lane) * 16 : p.x + min(8 * n + g, p.m - 1) * p.x_stride + t * (2 * kColumns);
  }
  wait_for_kernel_in_front();

  float part[MR][NT][4], sum[MR][NT][4];
#pragma unroll
  for (int i = 0; i < MR; ++i) {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int c = 0; c < 4; ++c) part[i][n][c] = sum[i][n][c] = 0.0f;
    }
  }
  const uint32_t base_x = (BF16 ? tile::kBf16Base * 0x10001u : 0x64006400u) ^ (p.nibble_xor & 0x000F000Fu);
  int until_flush = p.flush_steps - (s0 & (p.flush_steps - 1));
  // Two levels of sums: chains of four multiply-adds in registers, and the chains in the warp's own part of
  // `red`, so that a result is no further from float64 than those of the kernels for other batches
  // (int4, groups of 32, 4096 columns: one chain of 16 7.8e-8 of the result, tcgen05 kernel 6.6e-8, digits 8.1e-8).
  constexpr int kChain = 4;
  int chained = 0;
  bool begun = false;
  auto keep = [&]() {
#pragma unroll
    for (int i = 0; i < MR; ++i) {
#pragma unroll
      for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float& total = red[warp][16 * i + 8 * (c >> 1) + g][8 * n + 2 * t + (c & 1)];
          total = begun ? total + sum[i][n][c] : sum[i][n][c];
          sum[i][n][c] = 0.0f;
        }
      }
    }
    begun = true;
    chained = 0;
  };
  uint4 ahead[NT][kFrags];
  // 16 bytes of column tile n: eight columns of the lane
  auto load_x = [&](int step, int q, int plane, int n) {
    return load_activations(FRAGMENTS ? x_at[n] + ((step * kFrags + q) * PLANES + plane) * (NT * 512)
                                      : x_at[n] + step * (2 * STEP) + 16 * q);
  };
  auto fetch_x = [&](int step) {
    const bool inside = step < s1 && (FRAGMENTS || step * STEP + t * kColumns < p.columns);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int q = 0; q < kFrags; ++q) {
        ahead[n][q] = make_uint4(0u, 0u, 0u, 0u);
        if (inside) ahead[n][q] = load_x(step, q, 0, n);
      }
    }
  };
  if (kEarly) fetch_x(s0);
  for (int s = s0; s < s1; s += AHEAD) {
#pragma unroll
    for (int d = 0; d < AHEAD; ++d) {
      const int step = s + d;
      if (step < s1) {
        if (step * STEP >= boundary) {
          take_group();
          ++group;
          boundary += p.group;
          fetch_group(min(group + 1, p.groups - 1));
        }
        const bool inside = FRAGMENTS || step * STEP + t * kColumns < p.columns;
        uint4 early[NT][kFrags];
        if (kEarly) {
#pragma unroll
          for (int n = 0; n < NT; ++n) {
#pragma unroll
            for (int q = 0; q < kFrags; ++q) early[n][q] = ahead[n][q];
          }
          fetch_x(step + 1);
        }
        // eight columns of the lane, 32 of the quad, at a time
#pragma unroll
        for (int q = 0; q < kFrags; ++q) {
          uint32_t a[MR][2][4];
#pragma unroll
          for (int i = 0; i < MR; ++i) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if constexpr (kNibbles) {
                const uint4 v = FRAGMENTS ? tile::convert_nibbles_apart<BF16>(ring[d][i][h][q], base_x, base_z[i][h])
                                          : tile::convert_nibbles<BF16>(ring[d][i][h][q] ^ p.nibble_xor, base_z[i][h]);
                a[i][h][0] = v.x;
                a[i][h][1] = v.y;
                a[i][h][2] = v.z;
                a[i][h][3] = v.w;
              } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  a[i][h][k] = tile::convert_bytes2<BF16>(ring[d][i][h][2 * q + (k >> 1)], k & 1 ? 0x4342u : 0x4140u);
                }
              }
            }
          }
          if (q + 1 == kFrags && step + AHEAD < s1) fetch(ring[d], step + AHEAD);
#pragma unroll
          for (int plane = PLANES - 1; plane >= 0; --plane) {  // (the small parts first)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              uint4 b = make_uint4(0u, 0u, 0u, 0u);
              if (kEarly) {
                b = early[n][q];
              } else if (inside) {
                b = load_x(step, q, plane, n);
              }
#pragma unroll
              for (int i = 0; i < MR; ++i) {
                mma_f16<BF16>(part[i][n], a[i][0][0], a[i][1][0], a[i][0][1], a[i][1][1], b.x, b.y);
                mma_f16<BF16>(part[i][n], a[i][0][2], a[i][1][2], a[i][0][3], a[i][1][3], b.z, b.w);
              }
            }
          }
        }
        if (--until_flush == 0 || step + 1 == s1) {
          until_flush = p.flush_steps;
#pragma unroll
          for (int i = 0; i < MR; ++i) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                sum[i][n][c] = fmaf(part[i][n][c], scale[i][c >> 1], sum[i][n][c]);
                part[i][n][c] = 0.0f;
              }
            }
          }
          if (++chained == kChain) keep();
        }
      }
    }
  }
  if (chained != 0 || !begun) keep();
  __syncthreads();
  // the warps' parts of K are added in 64 bits, in order
  for (int i = threadIdx.x; i < kR * 8 * NT; i += kThreads) {
    const int r = i % kR, token = i / kR;
    const int row = row0 + r;
    if (row >= p.rows || token >= p.m) continue;
    double total = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) total += red[w][r][token];
    float out = static_cast<float>(total);
    if (p.bias != nullptr) out += __ldg(p.bias + row);
    if (p.activation != QX_ACTIVATION_NONE) out = projection_activation(out, p.activation);
    store_output(p.y, p.y_type, token * p.ldy + row, out);
  }
}

// ---- activations in front ----------------------------------------------------------------------
constexpr int kRowThreads = 512;

// max over the block of values that are never negative
__device__ __forceinline__ float block_max(float v, float* shared) {
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, h));
  if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = v;
  __syncthreads();
  v = shared[threadIdx.x & (kRowThreads / 32 - 1)];
#pragma unroll
  for (int h = kRowThreads / 64; h >= 1; h >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, h));
  return v;
}
__device__ __forceinline__ float storage_value(const void* x, int type, long long index) {
  if (type == QX_STORAGE_F32) return static_cast<const float*>(x)[index];
  const uint16_t bits = static_cast<const uint16_t*>(x)[index];
  return type == QX_STORAGE_F16 ? __half2float(__ushort_as_half(bits)) : __uint_as_float(static_cast<uint32_t>(bits) << 16);
}
// eight activations from `index` on, zero from `count` of them on
__device__ __forceinline__ void load_eight(const void* x, int type, long long index, long long count, bool vector,
                                           float (&v)[8]) {
  if (vector && count >= 8) {
    if (type == QX_STORAGE_F32) {
      const float4 a = *reinterpret_cast<const float4*>(static_cast<const float*>(x) + index);
      const float4 b = *reinterpret_cast<const float4*>(static_cast<const float*>(x) + index + 4);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
      const uint4 a = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + index);
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint16_t bits = static_cast<uint16_t>(w[i >> 1] >> (16 * (i & 1)));
        v[i] = type == QX_STORAGE_F16 ? __half2float(__ushort_as_half(bits))
                                      : __uint_as_float(static_cast<uint32_t>(bits) << 16);
      }
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = i < count ? storage_value(x, type, index + i) : 0.0f;
}

// One block per row. A thread's first kHeld groups of eight stay in registers between the two passes.
constexpr int kHeld = 2;
template <class Use>
__device__ __forceinline__ void for_groups(const void* x, int type, long long base, long long columns, long long groups,
                                           bool vector, float (&held)[kHeld][8], bool first, Use&& use) {
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const long long at = threadIdx.x + static_cast<long long>(i) * kRowThreads;
    if (at < groups) {
      if (first) load_eight(x, type, base + 8 * at, columns - 8 * at, vector, held[i]);
      use(at, held[i]);
    }
  }
  for (long long at = threadIdx.x + static_cast<long long>(kHeld) * kRowThreads; at < groups; at += kRowThreads) {
    float v[8];
    load_eight(x, type, base + 8 * at, columns - 8 * at, vector, v);
    use(at, v);
  }
}

// Where eight int8 activations from `column` on of column `c` of the product lie in the order in which
// the lanes read them: [step of 64][column tile][lane][16 columns].
__device__ __forceinline__ long long fragment_byte(long long c, long long column, int column_tiles) {
  const long long step = column / 64;
  const int lane = static_cast<int>(c & 7) * 4 + static_cast<int>(column / 16 & 3);
  return ((step * column_tiles + c / 8) * 32 + lane) * 16 + (column & 15);
}

// 16-bit activations in that order: [step][eight columns of a lane][plane][column tile][lane]; f32 ones as
// three bf16 planes, each the truncated remainder of the ones before, so that their sum is the value. `apart`: the eight
// columns as convert_nibbles_apart has them.
template <int PLANES>
__global__ void __launch_bounds__(256) stream_fragments_kernel(const void* __restrict__ x, int x_type,
                                                               const int* __restrict__ order, uint4* __restrict__ out,
                                                               int columns, int m, int lane_columns, int column_tiles,
                                                               int total, int vector, int apart) {
  launch_dependents();  // (the projection's weights are prepared ones)
  wait_for_kernel_in_front();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= total) return;
  const int lane = i & 31, n = i / 32 % column_tiles, piece = i / 32 / column_tiles;
  const int per_step = lane_columns / 8;
  const int token = 8 * n + (lane >> 2);
  const int column = (piece / per_step * 4 + (lane & 3)) * lane_columns + piece % per_step * 8;
  const int count = token < m ? columns - column : 0;
  const long long base = static_cast<long long>(token < m ? token : 0) * columns;
  uint32_t words[PLANES][4];
  if (PLANES == 1 && order == nullptr && vector != 0 && count >= 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + base + column);
    out[i] = apart != 0 ? make_uint4(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.x, v.z, 0x7632),
                                     __byte_perm(v.y, v.w, 0x5410), __byte_perm(v.y, v.w, 0x7632))
                        : v;
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int plane = 0; plane < PLANES; ++plane) words[plane][j] = 0u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = apart != 0 ? j + 4 * h : 2 * j + h;
      if (k < count) {
        const long long from = base + (order != nullptr ? order[column + k] : column + k);
        if (PLANES == 3) {
          float v = static_cast<const float*>(x)[from];
#pragma unroll
          for (int plane = 0; plane < PLANES; ++plane) {
            const uint32_t top = __float_as_uint(v) & 0xffff0000u;
            words[plane][j] |= h == 0 ? top >> 16 : top;
            v -= __uint_as_float(top);
          }
        } else {
          words[0][j] |= static_cast<uint32_t>(static_cast<const uint16_t*>(x)[from]) << (16 * h);
        }
      }
    }
  }
#pragma unroll
  for (int plane = 0; plane < PLANES; ++plane) {
    out[(static_cast<long long>(piece) * PLANES + plane) * (32 * column_tiles) + (i - piece * 32 * column_tiles)] =
        make_uint4(words[plane][0], words[plane][1], words[plane][2], words[plane][3]);
  }
}

__global__ void __launch_bounds__(kRowThreads) stream_codes_kernel(const float* __restrict__ x, int8_t* __restrict__ codes,
                                                                   float* __restrict__ scales, int* __restrict__ sums,
                                                                   long long columns, long long stride, int column_tiles, int vector) {
  // (the GEMM behind reads nothing of its caller's before it has waited for this kernel)
  launch_dependents();
  wait_for_kernel_in_front();
  __shared__ float warp_max[kRowThreads / 32];
  __shared__ int warp_sum[kRowThreads / 32];
  const long long row = blockIdx.x, base = row * columns;
  const long long groups = stride / 8;
  float held[kHeld][8];
  float maximum = 0.0f;
  for_groups(x, QX_STORAGE_F32, base, columns, groups, vector != 0, held, true, [&](long long, const float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) maximum = fmaxf(maximum, fabsf(v[i]));
  });
  maximum = block_max(maximum, warp_max);
  const float scale = __fdiv_rn(maximum, 127.0f);
  const float inverse = scale > 0.0f ? __fdiv_rn(1.0f, scale) : 0.0f;
  int sum = 0;
  for_groups(x, QX_STORAGE_F32, base, columns, groups, vector != 0, held, false, [&](long long at, const float (&v)[8]) {
    uint32_t word[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int q = max(-127, min(127, __float2int_rn(__fmul_rn(v[i], inverse))));
      word[i & 1] |= static_cast<uint32_t>(q & 255) << (8 * (i >> 1));
      sum += q;
    }
    *reinterpret_cast<uint2*>(codes + fragment_byte(row, 8 * at, column_tiles)) = make_uint2(word[0], word[1]);
  });
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, h);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
#pragma unroll
    for (int w = 0; w < kRowThreads / 32; ++w) total += warp_sum[w];
    scales[row] = scale;
    sums[row] = total;
  }
}

// The whole number nearest to t, for any t below 2^31 (the conversion unit, at 16 a cycle, would bound the kernel).
__device__ __forceinline__ float nearest_whole(float t) {
  const float s = copysignf(8388608.0f, t);  // (2^23: from there on t has no fraction)
  return fabsf(t) < 8388608.0f ? __fsub_rn(__fadd_rn(t, s), s) : t;
}
// The four balanced base-256 digits of each of four numbers, as four words of one digit each.
__device__ __forceinline__ void digit_words(const int (&t)[4], uint32_t (&word)[4]) {
  uint32_t v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = (static_cast<uint32_t>(t[i]) + 0x00808080u) ^ 0x00808080u;
  const uint32_t low01 = __byte_perm(v[0], v[1], 0x5140), low23 = __byte_perm(v[2], v[3], 0x5140);
  const uint32_t high01 = __byte_perm(v[0], v[1], 0x7362), high23 = __byte_perm(v[2], v[3], 0x7362);
  word[0] = __byte_perm(low01, low23, 0x5410);
  word[1] = __byte_perm(low01, low23, 0x7632);
  word[2] = __byte_perm(high01, high23, 0x5410);
  word[3] = __byte_perm(high01, high23, 0x7632);
}

// DIGITS rows per token: 4, or 8 with the remainders of the first four in the last. digit_ctas() CTAs per token: each takes
// the maxima over the whole row and writes its share of the digits, so that no SM converts a row alone (one token, both
// launches on 4096 x 4096, weights from memory: 7.0 us with four; 16 tokens 11.6 with two, 11.8 with four).
constexpr int digit_ctas(int digits) { return digits == 8 ? 4 : 2; }
template <int DIGITS>
__global__ void __launch_bounds__(kRowThreads) stream_digits_kernel(const void* __restrict__ x, int x_type,
                                                                    int8_t* __restrict__ digits, float* __restrict__ e_out,
                                                                    long long columns, int column_tiles, int vector) {
  launch_dependents();  // (the projection's weights are prepared ones)
  wait_for_kernel_in_front();
  __shared__ float warp_max[kRowThreads / 32], warp_least[kRowThreads / 32], warp_rest[kRowThreads / 32];
  constexpr int kDigitCtas = digit_ctas(DIGITS);
  const long long token = blockIdx.x / kDigitCtas, base = token * columns;
  const int share = blockIdx.x % kDigitCtas;
  const long long groups = (columns + 63) / 64 * 8;  // (whole steps)
  const float infinity = __uint_as_float(0x7f800000u);
  float held[kHeld][8];
  float amax = 0.0f, least = infinity;  // of the row; of the largest of any eight columns that are not all zero
  for_groups(x, x_type, base, columns, groups, vector != 0, held, true, [&](long long, const float (&v)[8]) {
    float largest = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // (fmaxf drops a NaN)
      const float a = fabsf(v[i]);
      largest = a < infinity ? fmaxf(largest, a) : infinity;
    }
    amax = fmaxf(amax, largest);
    if (DIGITS == 8 && largest > 0.0f) least = fminf(least, largest);
  });
  if (DIGITS == 8) {
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) least = fminf(least, __shfl_xor_sync(0xffffffffu, least, h));
    if ((threadIdx.x & 31) == 0) warp_least[threadIdx.x >> 5] = least;
  }
  amax = block_max(amax, warp_max);  // (and its barrier)
  // envelope 2^E > amax, t = x * 2^30 / 2^E; four digits: an activation below 2^-100 counts as zero
  auto exponent = [](float maximum) {
    const int biased = static_cast<int>(__float_as_uint(maximum) >> 23) + 1;
    return biased < 58 ? 58 : biased;
  };
  auto fixed = [](int biased) { return __uint_as_float(static_cast<uint32_t>(284 - biased) << 23); };
  const int biased = exponent(amax);
  const bool finite = biased < 256;
  const float to_fixed = finite ? fixed(biased) : 0.0f;
  auto scaled = [&](float v) { return finite ? __fmul_rn(v, to_fixed) : 0.0f; };
  // A remainder is at most a half. Under that envelope eight columns keep the 23 bits that they would have under their
  // own down to 2^-39 of the row's; a row with smaller ones beside its largest takes the largest remainder's envelope.
  int rest_biased = 127;
  if (DIGITS == 8) {
#pragma unroll
    for (int w = 0; w < kRowThreads / 32; ++w) least = fminf(least, warp_least[w]);
    if (least < __uint_as_float(static_cast<uint32_t>(finite ? biased - 39 : 1) << 23)) {
      float rmax = 0.0f;
      for_groups(x, x_type, base, columns, groups, vector != 0, held, false, [&](long long, const float (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float t = scaled(v[i]);
          rmax = fmaxf(rmax, fabsf(__fsub_rn(t, nearest_whole(t))));  // (exact)
        }
      });
      rest_biased = exponent(block_max(rmax, warp_rest));
    }
  }
  const float rest_fixed = fixed(rest_biased);
  for_groups(x, x_type, base, columns, groups, vector != 0, held, false, [&](long long at, const float (&v)[8]) {
    if ((at / 32) % kDigitCtas != share) return;  // (a warp's groups together)
#pragma unroll
    for (int half = 0; half < DIGITS / 4; ++half) {
      uint32_t word[2][4];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        int whole[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float t = scaled(v[4 * q + i]);
          whole[i] = __float2int_rn(half == 0 ? t : __fmul_rn(__fsub_rn(t, nearest_whole(t)), rest_fixed));
        }
        digit_words(whole, word[q]);
      }
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        *reinterpret_cast<uint2*>(digits + fragment_byte(DIGITS * token + 4 * half + d, 8 * at, column_tiles)) =
            make_uint2(word[0][d], word[1][d]);
      }
    }
  });
  if (threadIdx.x == 0 && share == 0) {
    const float e = finite ? __uint_as_float(static_cast<uint32_t>(biased - 30) << 23) : __uint_as_float(0x7fc00000u);
    if (DIGITS == 8) {
      e_out[2 * token] = e;
      e_out[2 * token + 1] = __uint_as_float(static_cast<uint32_t>(rest_biased - 30) << 23);
    } else {
      e_out[token] = e;
    }
  }
}

template <class... Params, class... Args>
qx_status launch(void (*kernel)(Params...), long long grid, int block, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attribute{};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(static_cast<unsigned>(grid));
  config.blockDim = dim3(static_cast<unsigned>(block));
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = 1;
  QX_CUDA_TRY(cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...));
  count_launch();
  return QX_STATUS_OK;
}

// Weight rows per warp: two tiles of 16 (every B fragment then feeds two MMAs) where CTAs of one tile would be more than
// two per SM, the third of which finds the SM full; one tile and more CTAs below that. Measured (us, two tiles | one): 8192 x
// 4096: int8 digits of 4 tokens 13.0 | 18.7, W8A8 16 rows 10.5 | 14.6, uint4 8 tokens 10.7 | 13.2;  5120 x 5120: digits of 2
// tokens 11.8 | 17.0, W8A8 16 rows 11.2 | 16.2, uint4 8 tokens 12.2 | 14.3, 16 tokens 14.3 | 16.6, W4A8 32 rows 14.4 | 20.7;
// 4096 x 4096: uint4 8 tokens 9.2 | 6.3, W8A8 24 rows 10.2 | 7.6.
constexpr long long kWideRows = 2 * 148 * 16 + 1;
// One column tile of whole numbers has registers for three CTAs, and nibbles with two tiles one round more of them: digits of
// one token 5120 x 5120 10.5 | 9.0, W4A8 16 rows 11.7 | 10.8.
constexpr long long kWideRowsOfFew = 32 * 192;

int prefetched_rows(long long row_bytes, long long rows, long long of_more) {
  return static_cast<int>(row_bytes * rows <= kPrefetchWhole ? rows : of_more / row_bytes);
}

int column_tiles(long long columns) { return columns <= 8 ? 1 : (columns <= 16 ? 2 : (columns <= 32 ? 4 : 8)); }

template <StreamSource SRC, bool FRAGMENTS, int NT>
qx_status launch_int(const IntParams& p, cudaStream_t stream) {
  // Eight column tiles: one CTA per SM either way, and rows on any byte have no registers for two tiles of
  // rows (40 tokens on 14336 x 8190 68 us against 91). Four of W8A8 come with up to 4096 rows only.
  constexpr bool kOne = SRC == kStreamNibblesLoose ? NT == 8 : (SRC == kStreamBytes && !FRAGMENTS && NT == 4);
  constexpr bool kTwo = NT == 8 && SRC != kStreamNibblesLoose;
  constexpr long long kWide = NT == 1 || (NT == 2 && SRC != kStreamBytes) ? kWideRowsOfFew : kWideRows;
  if constexpr (!kOne) {
    if (kTwo || p.rows >= kWide) {
      return launch(stream_int_kernel<SRC, FRAGMENTS, NT, 2, (NT <= 2 && SRC == kStreamNibbles ? 4 : 2), (NT == 8 ? 1 : 2)>,
                    (p.rows + 31) / 32, kThreads, stream, p);
    }
  }
  if constexpr (!kTwo) {
    return launch(stream_int_kernel<SRC, FRAGMENTS, NT, 1, (NT == 8 ? 2 : 4), (NT == 8 ? 1 : (NT == 1 ? 3 : 2))>,
                  (p.rows + 15) / 16, kThreads, stream, p);
  }
}
template <StreamSource SRC, bool FRAGMENTS>
qx_status launch_int(const IntParams& p, cudaStream_t stream) {
  static_assert(kStreamW8A8Rows <= 32);
  switch (column_tiles(p.x_rows)) {
    case 1: return launch_int<SRC, FRAGMENTS, 1>(p, stream);
    case 2: return launch_int<SRC, FRAGMENTS, 2>(p, stream);
    case 4: return launch_int<SRC, FRAGMENTS, 4>(p, stream);
    default: return launch_int<SRC, FRAGMENTS, SRC == kStreamBytes && !FRAGMENTS ? 4 : 8>(p, stream);
  }
}

template <StreamSource SRC, bool FRAGMENTS, bool BF16, int PLANES, int STEP, int NT>
qx_status launch_scaled(const ScaledParams& p, cudaStream_t stream) {
  constexpr bool kRoom = NT <= 2 && PLANES == 1;  // registers for two tiles of rows
  if constexpr (kRoom) {
    if (p.rows >= kWideRows) {
      return launch(stream_scaled_kernel<SRC, FRAGMENTS, BF16, PLANES, STEP, NT, 2, 2, 2>, (p.rows + 31) / 32, kThreads,
                    stream, p);
    }
  }
  return launch(stream_scaled_kernel<SRC, FRAGMENTS, BF16, PLANES, STEP, NT, 1, 4, 2>, (p.rows + 15) / 16, kThreads,
                stream, p);
}
template <StreamSource SRC, bool BF16, int PLANES, int STEP>
qx_status launch_scaled(const ScaledParams& p, bool fragments, cudaStream_t stream) {
  if (!fragments) return launch_scaled<SRC, false, BF16, 1, STEP, 1>(p, stream);  // (one column tile of 16-bit rows)
  if (p.m <= 8) return launch_scaled<SRC, true, BF16, PLANES, STEP, 1>(p, stream);
  if (p.m <= 16) return launch_scaled<SRC, true, BF16, PLANES, STEP, 2>(p, stream);
  return launch_scaled<SRC, true, BF16, PLANES, STEP, 4>(p, stream);
}
template <StreamSource SRC>
qx_status launch_scaled(const ScaledParams& p, bool bf16, int planes, int step, bool fragments, cudaStream_t stream) {
  if (planes == 3) {
    return step == 32 ? launch_scaled<SRC, true, 3, 32>(p, fragments, stream)
                      : launch_scaled<SRC, true, 3, 64>(p, fragments, stream);
  }
  if (bf16) {
    return step == 32 ? launch_scaled<SRC, true, 1, 32>(p, fragments, stream)
                      : launch_scaled<SRC, true, 1, 64>(p, fragments, stream);
  }
  if (SRC == kStreamBytes || step == 32) return launch_scaled<SRC, false, 1, 32>(p, fragments, stream);
  return launch_scaled<kStreamNibbles, false, 1, 64>(p, fragments, stream);
}

// columns whose sum leaves the tensor core (the limits of qx_scaled_gemm.cu)
int promote_columns(const StreamScaledArgs& a) {
  const int planes = a.x_type == QX_STORAGE_F32 ? 3 : 1;
  int promote = a.group % 128 == 0 || a.group == a.columns ? 128 : (a.group % 64 == 0 ? 64 : 32);
  if (planes == 3 && promote > 64) promote = 64;
  if (a.source == kStreamBytes && a.x_type == QX_STORAGE_F16) promote = 32;
  return promote;
}
int step_columns(const StreamScaledArgs& a) { return promote_columns(a) == 32 ? 32 : 64; }
// Whether the activations are laid out for the lanes in front: f32 and gathered ones, rows off 16 bytes,
// and more than one column tile (the lanes' reads of plain rows touch eight lines each, and
// L1 is what bounds a warp of two tiles and more).
bool wants_fragments(const StreamScaledArgs& a) {
  return a.x_type == QX_STORAGE_F32 || a.order != nullptr || a.m > 8 || reinterpret_cast<uintptr_t>(a.x) % 16 != 0;
}

}  // namespace

bool stream_int_serves(const StreamIntArgs& a) {
  const int most = a.result == kStreamW8A8 ? kStreamW8A8Rows : kStreamColumns;
  if (a.x_rows < 1 || a.x_rows > most || a.rows < 1 || a.rows > (1LL << 30) || a.columns > 131000) return false;
  if (reinterpret_cast<uintptr_t>(a.x) % 16 != 0) return false;
  if (a.source == kStreamBytes) return a.columns % 16 == 0 && reinterpret_cast<uintptr_t>(a.codes) % 16 == 0;
  return a.source == kStreamNibblesLoose || (a.columns % 16 == 0 && reinterpret_cast<uintptr_t>(a.codes) % 8 == 0);
}

qx_status launch_stream_int(const StreamIntArgs& a, cudaStream_t stream) {
  IntParams p{};
  p.codes = a.codes;
  p.row_bytes = a.source == kStreamBytes ? a.columns : (a.columns + 1) / 2;
  p.codes_end = a.codes + p.row_bytes * a.rows;
  p.x = reinterpret_cast<const uint8_t*>(a.x);
  p.ws = a.ws;
  p.as = a.as;
  p.row_sum = a.row_sum;
  p.zp = a.zp;
  p.bias = a.bias;
  p.y = a.y;
  p.acc = a.acc;
  p.x_stride = a.columns;
  p.ldy = a.ldy;
  p.rows = static_cast<int>(a.rows);
  p.columns = static_cast<int>(a.columns);
  p.x_rows = a.x_rows;
  p.steps = static_cast<int>((a.columns + 63) / 64);
  p.activation = a.activation;
  p.y_type = a.y_type;
  p.prepared = a.prepared ? 1 : 0;
  p.prefetch_rows = prefetched_rows(p.row_bytes, a.rows, kPrefetchFirst);
  p.digits = a.digits;
  switch (a.source) {
    case kStreamBytes:
      return a.result == kStreamDigits ? launch_int<kStreamBytes, true>(p, stream)
                                       : launch_int<kStreamBytes, false>(p, stream);
    case kStreamNibbles: return launch_int<kStreamNibbles, true>(p, stream);
    default: return launch_int<kStreamNibblesLoose, true>(p, stream);
  }
}

size_t stream_code_bytes(long long x_rows, long long columns) {
  return static_cast<size_t>((columns + 63) / 64) * 512 * column_tiles(x_rows);
}
qx_status launch_stream_codes(const float* x, int8_t* codes, float* scales, int* sums, long long m, long long columns,
                              cudaStream_t stream) {
  const int vector = columns % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 ? 1 : 0;
  return launch(stream_codes_kernel, m, kRowThreads, stream, x, codes, scales, sums, columns,
                (columns + 63) / 64 * 64, column_tiles(m), vector);
}
qx_status launch_stream_digits(const void* x, int x_type, int8_t* digits, float* e, long long m, long long columns,
                               int per_token, cudaStream_t stream) {
  const int vector = reinterpret_cast<uintptr_t>(x) % 16 == 0 ? 1 : 0;
  return launch(per_token == 8 ? stream_digits_kernel<8> : stream_digits_kernel<4>, digit_ctas(per_token) * m, kRowThreads,
                stream, x, x_type, digits, e, columns, column_tiles(per_token * m), vector);
}

bool stream_scaled_serves(const StreamScaledArgs& a) {
  if (a.m < 1 || a.m > 32 || a.rows < 1 || a.rows > (1LL << 30) || a.columns > (1LL << 24)) return false;
  if (a.columns % 16 != 0 || reinterpret_cast<uintptr_t>(a.codes) % 16 != 0) return false;
  return a.group == a.columns || a.group % 32 == 0;
}

size_t stream_scaled_scratch_bytes(const StreamScaledArgs& a) {
  if (!wants_fragments(a)) return 0;
  const size_t steps = static_cast<size_t>((a.columns + step_columns(a) - 1) / step_columns(a));
  return steps * step_columns(a) * (a.x_type == QX_STORAGE_F32 ? 6 : 2) * 8 * column_tiles(a.m);
}

qx_status launch_stream_scaled(const StreamScaledArgs& a, void* scratch, cudaStream_t stream) {
  const int step = step_columns(a), planes = a.x_type == QX_STORAGE_F32 ? 3 : 1;
  const bool fragments = wants_fragments(a);
  ScaledParams p{};
  p.steps = static_cast<int>((a.columns + step - 1) / step);
  p.x = static_cast<const uint8_t*>(fragments ? scratch : a.x);
  if (fragments) {
    const int tiles = column_tiles(a.m), total = p.steps * (step / 32) * tiles * 32;
    const int vector = a.columns % 8 == 0 && reinterpret_cast<uintptr_t>(a.x) % 16 == 0 ? 1 : 0;
    QX_TRY(launch(planes == 3 ? stream_fragments_kernel<3> : stream_fragments_kernel<1>, (total + 255) / 256, 256, stream,
                  a.x, a.x_type, a.order, static_cast<uint4*>(scratch), static_cast<int>(a.columns),
                  static_cast<int>(a.m), step / 4, tiles, total, vector, a.source == kStreamNibbles ? 1 : 0));
  }
  p.codes = a.codes;
  p.scales = a.scales;
  p.zeros = a.zeros;
  p.bias = a.bias;
  p.y = a.y;
  p.row_bytes = a.source == kStreamBytes ? a.columns : a.columns / 2;
  p.x_stride = a.columns * 2;
  p.ldy = a.ldy;
  p.nibble_xor = a.nibble_xor;
  p.rows = static_cast<int>(a.rows);
  p.columns = static_cast<int>(a.columns);
  p.m = static_cast<int>(a.m);
  p.group = static_cast<int>(a.group);
  p.groups = static_cast<int>(a.columns / a.group);
  p.activation = a.activation;
  p.y_type = a.y_type;
  p.flush_steps = promote_columns(a) / step;
  p.prefetch_rows = prefetched_rows(p.row_bytes, a.rows, 0);
  const bool bf16 = a.x_type != QX_STORAGE_F16;
  return a.source == kStreamBytes ? launch_scaled<kStreamBytes>(p, bf16, planes, step, fragments, stream)
                                  : launch_scaled<kStreamNibbles>(p, bf16, planes, step, fragments, stream);
}

}  // namespace qx
