// Pieces of the persistent tensor-core kernel whose weights are converted to 16-bit operands on
// the way (qx_scaled_gemm.cu): ring positions, bulk copies, packed f32 arithmetic and the exact
// conversions of integer codes.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "qx_sm100.cuh"

namespace qx {
namespace tile {

struct Ring {
  uint32_t slot = 0, phase = 0;
  __device__ __forceinline__ void advance(uint32_t slots) {
    if (++slot == slots) {
      slot = 0;
      phase ^= 1u;
    }
  }
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(sm100::smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(sm100::smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void wait_for_kernel_in_front() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---- two f32 values in a 64-bit register -------------------------------------------------
__device__ __forceinline__ unsigned long long pack2(uint32_t lo, uint32_t hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}
__device__ __forceinline__ void unpack2(unsigned long long v, uint32_t& lo, uint32_t& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ unsigned long long addf2(unsigned long long a, unsigned long long b) {
  unsigned long long v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ unsigned long long subf2(unsigned long long a, unsigned long long b) {
  unsigned long long v;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
// total += value; what the rounding of that lost goes to `rest` (Dekker's fast two-sum: exact where
// the total is the larger one, as it is of a sum of many, and at worst one more rounding of a value)
__device__ __forceinline__ void add_with_rest2(unsigned long long& total, unsigned long long& rest,
                                               unsigned long long value) {
  const unsigned long long sum = addf2(total, value);
  rest = addf2(rest, subf2(value, subf2(sum, total)));
  total = sum;
}

// ---- 16-bit whole numbers ----------------------------------------------------------------
// bf16 ones carry 2^-16: a group's sum of bf16 activations of any size then stays finite in f32
// (2^128 * 2^8 * 128 columns * 2^-16), and no bit of a normal activation's product falls below
// 2^-149. The scales carry 2^16 in return. f16 activations are small enough as they are.
constexpr float kBf16Unscale = 65536.0f;
constexpr uint32_t kBf16Base = 0x3B00u;  // 128 * 2^-16: unit steps of 2^-16

template <bool BF16>
__device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
  if (BF16) {
    const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a),
                                     *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Two signed bytes of `w` picked by `selector` (its upper bytes take byte 4) -> two 16-bit whole
// numbers.
template <bool BF16>
__device__ __forceinline__ uint32_t convert_bytes2(uint32_t w, uint32_t selector) {
  if (BF16) {
    // (128 + low seven bits) - (128, or 256 for a negative code), all times 2^-16
    const uint32_t p = __byte_perm(w, kBf16Base >> 8, selector);
    return sub2<true>(p & 0xFF7FFF7Fu, p & 0xFF80FF80u);
  }
  // code ^ 0x80 = code + 128 under the exponent of 1024
  const uint32_t p = __byte_perm(w ^ 0x80808080u, 0x64646464u, selector);
  return sub2<false>(p, 0x64806480u);
}

// Eight nibbles -> eight 16-bit whole numbers nibble - z in column order. A nibble under the
// exponent bits of `magic` (f16 1024 = 0x6400, bf16 128 times 2^-16: steps of one) is base + nibble;
// `base_z` holds base + z twice.
template <bool BF16>
__device__ __forceinline__ uint4 convert_nibbles(uint32_t w, uint32_t base_z) {
  const uint32_t magic = BF16 ? kBf16Base * 0x10001u : 0x64006400u;
  const uint32_t high = w >> 4;
  uint32_t out[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t pair = __byte_perm(w, high, i | (i << 4) | ((4 + i) << 8) | ((4 + i) << 12));
    out[i] = sub2<BF16>((pair & 0x000F000Fu) | magic, base_z);
  }
  return make_uint4(out[0], out[1], out[2], out[3]);
}
// The same in the order (0, 4), (1, 5), (2, 6), (3, 7), which needs no byte permutes (those run at half rate);
// `base_x` is the base's bits with the nibbles' exclusive-or in them, twice.
template <bool BF16>
__device__ __forceinline__ uint4 convert_nibbles_apart(uint32_t w, uint32_t base_x, uint32_t base_z) {
  return make_uint4(sub2<BF16>((w & 0x000F000Fu) ^ base_x, base_z), sub2<BF16>(((w >> 4) & 0x000F000Fu) ^ base_x, base_z),
                    sub2<BF16>(((w >> 8) & 0x000F000Fu) ^ base_x, base_z),
                    sub2<BF16>(((w >> 12) & 0x000F000Fu) ^ base_x, base_z));
}
// z as it is subtracted: (base + z) twice
template <bool BF16>
__device__ __forceinline__ uint32_t zero_word(float z) {
  uint32_t bits;
  if (BF16) {
    bits = __float_as_uint((128.0f + z) / kBf16Unscale) >> 16;  // exact: 128 .. 143
  } else {
    bits = __half_as_ushort(__float2half_rn(1024.0f + z));
  }
  return bits | (bits << 16);
}

}  // namespace tile
}  // namespace qx
