// Batched projections with weight scales along K on the tensor cores:
//   Y[t, o] = act( sum_g s[o, g] * sum_{k in g} (q[o, k] - z[o, g]) * x[t, k]  + bias[o] )
// for canonical nibbles / bytes with group scales (qgemm_prepacked_epilogue_storage,
// kernels/quantization/qgemm_canonical.cpp:4460-4648) and q8_0 blocks with bf16 activations
// (qgemm_prepacked, qgemm_panel.cpp:214-287).
//
// Arithmetic. The codes minus their zero point are whole numbers of at most eight bits, exact
// in f16 and in bf16, and the activations enter in their own 16-bit type (f32 activations as
// three bf16 planes whose sum is the value, multiplied one after the other into the same
// accumulator). So every product is exact, a group's sum is formed by the tensor core in f32
// over at most 128 columns, and the f32 scale is applied once per group by an f32 multiply-add
// on the CUDA cores: no scale is ever rounded to 16 bits. Whole numbers in bf16 carry 2^-16, so
// that no group's sum leaves the range of f32. (f32 tokens that are below 2^-110 altogether lose
// low bits: their third plane is below the smallest bf16.)
//
// Pipeline (persistent CTAs, one per SM, 28 warps):
//   warp 0       packed codes: 16 KiB slots of [128 rows][128 bytes], 128-byte swizzled
//                (256 columns of nibbles, 128 of bytes), by TMA or, from a panel, bulk copies
//   warp 2       activations: TMA tiles of bn tokens x 64 columns, into the stage's B part
//   conv warps   thread = weight row: codes -> 16-bit whole numbers, into the stage's A part
//   warp 1       MMA issuer: one wait and one commit per stage (128 columns, all planes),
//                8 x tcgen05.mma per plane; a new accumulator every `promote` columns (32 / 64 /
//                128: what the group size allows)
//   epilogue     thread = weight row: tcgen05.ld, acc += scale * partial (packed f32x2 FMAs), every
//                8 or 16 of them into totals in TMEM; at the end bias, activation, store
// What bounds it is less the tensor core than the chains of single instructions around it: a
// successful barrier wait costs about 80 cycles, a commit 30, a pair of MMAs 100 or more, so a
// step of 64 columns with four waits and three commits took 1300 cycles where its MMAs (32
// tokens) take 150. Hence one barrier pair per stage for both operands and stages of 128
// columns. A converter or epilogue warp is such a chain as well (500 to 1000 cycles per 64
// columns): eight of each, and tiles of at most 128 tokens, whose accumulators leave registers
// for them (256 tokens with four converter warps: 163 us on 14336 x 4096 uint4 x 512 tokens).
//
// Work split. Whole tiles round robin when they fill the SMs, else the (tile, 256-column slab)
// sequence is cut into one contiguous range per CTA; pieces of a tile go to scratch memory and
// whoever completes a tile's count adds them in CTA order (nobody waits).

#include <cuda.h>

#include "qx_gemv.cuh"
#include "qx_scaled_gemm.cuh"
#include "qx_sm100.cuh"
#include "qx_tile_pipe.cuh"

namespace qx {
namespace {

using namespace sm100;
using namespace tile;

constexpr int kRows = 128;                 // weight rows per tile
constexpr int kSub = 64;                   // columns of one operand sub-tile (128 bytes of 16 bits)
constexpr int kRawBytes = 16 * 1024;
// rows on any byte: nine 16-byte pieces from the boundary below a row's first byte on
constexpr int kLoosePitch = 9 * 16;
constexpr int kLooseBytes = kRows * kLoosePitch;
constexpr int raw_bytes(int source) { return source == kScaledNibblesLoose ? kLooseBytes : kRawBytes; }
constexpr int kABytes = kRows * 128;       // one converted sub-tile
constexpr int kSubs = 2;                   // operand sub-tiles per stage
constexpr int kStepCols = kSubs * kSub;
constexpr int kMaxStages = 3, kMaxRaw = 4, kMaxAcc = 4;
constexpr int kFinishCols = 16;            // columns an epilogue warp finishes at a time
constexpr size_t kSmemMax = 227 * 1024;
constexpr int kTmemCols = 512;             // all of it: one CTA per SM
// Scaled units in a row of f32 multiply-adds: rows of many units may take longer chains, as the digit
// kernels' own error grows with the row (q8_0: 6.6e-8 of the result at 32 units, 9.0e-8 at 256,
// 9.6e-8 at 344; chains of 8 are worth 6.2e-8 and chains of 16 8.0e-8 at any length).
constexpr int kChain = 8, kLongChain = 16, kLongRowUnits = 256;

// EPI epilogue warps, CONV converter warps, COLS accumulator columns of an epilogue warp at most.
// Registers per thread of the warpgroups (issue warps, epilogue, converters): they add up to at
// most what the block is launched with (checked against the compiled kernel in launch_kernel). With
// 32 for the issue warps the MMA thread spills (16 tokens on 14336 x 4096 uint4: 35.2 us against 31.6).
template <int EPI_, int CONV_, int COLS_, int RAW_, int R_ISSUE, int R_EPI, int R_CONV>
struct Shape {
  static constexpr int kEpi = EPI_, kConv = CONV_, kCols = COLS_, kRawSlots = RAW_;
  static constexpr int kThreads = 32 * (4 + EPI_ + CONV_);
  static constexpr int kGroups = CONV_ / 8;  // groups of eight converter warps take stages in turn
  static constexpr int kIssueRegs = R_ISSUE, kEpiRegs = R_EPI, kConvRegs = R_CONV;
  static constexpr int kRegShares = R_ISSUE + EPI_ / 4 * R_EPI + CONV_ / 4 * R_CONV;
  static constexpr int kTokens = COLS_ * (EPI_ / 4);  // per tile at most
  static constexpr int kFinishBytes = EPI_ * 32 * kFinishCols * 4;
  static_assert(COLS_ == 32, "an epilogue warp reads the columns of a unit at once");
  static_assert(RAW_ <= kMaxRaw && EPI_ <= kScaledEpilogueWarps && CONV_ % 8 == 0 &&
                    65536 / kThreads / 8 * 8 * (kThreads / 128) >= kRegShares, "shape");
};
using Small = Shape<8, 16, 32, 4, 40, 104, 56>;
using SmallPlanes = Shape<8, 16, 32, 2, 40, 104, 56>;  // three planes: larger stages
using Large = Shape<16, 8, 32, 3, 40, 88, 56>;

struct ScaledParams {
  const uint8_t* panel;
  const float* scales;
  const float* zeros;
  const float* bias;
  const float* token_scales;
  void* y;
  float* partial;
  int* counters;
  int* error;
  long long ldy, units, row_bytes, code_bytes;
  uint32_t nibble_xor;
  int m, rows, group, groups;
  int columns;                 // rounded up to whole stages
  int slabs, bn, stages;
  int promote, promote_log;    // columns per accumulator
  int hand_cols;               // columns per hand-over to the epilogue: promote .. a stage's
  int accs;                    // hand-overs in flight in TMEM
  int chain;                   // units per chain
  int o_tiles, r_tiles, split, y_type, activation;
};

struct __align__(16) ScaledBarriers {
  uint64_t raw_full[kMaxRaw], raw_empty[kMaxRaw];
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t tmem_full[kMaxAcc], tmem_empty[kMaxAcc];
  uint32_t tmem_base;
  int abort_flag;
};

template <class S>
constexpr size_t stage_bytes(int bn, int planes) {
  return static_cast<size_t>(kSubs) * (kABytes + static_cast<size_t>(planes) * bn * 128);
}
template <class S>
constexpr size_t other_bytes(int raw = kRawBytes) {
  return 1024 + S::kRawSlots * raw + S::kFinishBytes + sizeof(ScaledBarriers);
}
template <class S>
constexpr int stages_for(int bn, int planes, int raw = kRawBytes) {
  const size_t fit = (kSmemMax - other_bytes<S>(raw)) / stage_bytes<S>(bn, planes);
  return fit > kMaxStages ? kMaxStages : static_cast<int>(fit);
}
static_assert(stages_for<Small>(64, 1, kLooseBytes) >= 2 && stages_for<SmallPlanes>(64, 3) >= 2 &&
                  stages_for<Large>(128, 1, kLooseBytes) >= 2, "stages");

// Slabs [s0, s1) of 256 columns of a tile. Every role walks the same sequence.
struct Piece {
  int tile, s0, s1;
};
struct Walk {
  int u, end, slabs, split;
  __device__ explicit Walk(const ScaledParams& p) {
    slabs = p.slabs;
    split = p.split;
    if (split) {
      u = static_cast<int>(p.units * blockIdx.x / gridDim.x);
      end = static_cast<int>(p.units * (blockIdx.x + 1) / gridDim.x);
    } else {
      u = blockIdx.x;
      end = p.o_tiles * p.r_tiles;
    }
  }
  __device__ bool next(Piece& w) {
    if (u >= end) return false;
    if (split) {
      w.tile = u / slabs;
      w.s0 = u - w.tile * slabs;
      w.s1 = min(slabs, w.s0 + end - u);
      u += w.s1 - w.s0;
    } else {
      w.tile = u;
      w.s0 = 0;
      w.s1 = slabs;
      u += gridDim.x;
    }
    return true;
  }
};

template <int SRC, bool BF16, int PLANES, class S>
__global__ void __launch_bounds__(S::kThreads, 1)
scaled_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                   const ScaledParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const uint32_t b_sub = static_cast<uint32_t>(p.bn) * 128u;  // bn x 64 columns
  constexpr uint32_t kStageA = kSubs * kABytes;
  const uint32_t b_bytes = kSubs * PLANES * b_sub;
  const uint32_t stage_size = kStageA + b_bytes;
  uint8_t* raw_ring = smem + p.stages * stage_size;
  float* finish = reinterpret_cast<float*>(raw_ring + S::kRawSlots * raw_bytes(SRC));
  auto* bars = reinterpret_cast<ScaledBarriers*>(reinterpret_cast<uint8_t*>(finish) + S::kFinishBytes);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  volatile int* abort_flag = &bars->abort_flag;
  // columns of packed codes in one 16 KiB slot
  constexpr bool kLoose = SRC == kScaledNibblesLoose;
  constexpr bool kNibbles = SRC == kScaledNibbles || kLoose;
  constexpr int kRawCols = kNibbles ? 256 : 128;
  constexpr int kRaw = raw_bytes(SRC);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kRawSlots; ++s) {
      mbar_init(&bars->raw_full[s], kLoose ? 64 : 1);
      mbar_init(&bars->raw_empty[s], kNibbles ? S::kConv : 8);  // (a slot of bytes is one stage)
    }
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(&bars->full[s], 8 + 1);  // eight converter warps, activation copies
      mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < kMaxAcc; ++a) {
      mbar_init(&bars->tmem_full[a], 1);
      mbar_init(&bars->tmem_empty[a], S::kEpi);
    }
    bars->abort_flag = 0;
    mbar_fence_init();
    if (SRC != kScaledPanelQ8 && !kLoose) prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_x);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  asm volatile("griddepcontrol.launch_dependents;");
  Walk walk(p);
  Piece w;
  bool ok = true;
  int role = 0;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::kIssueRegs));
    if (kLoose && (warp == 0 || warp == 3)) {
      // ------------------------------ packed codes, rows on any byte ------------
      // Two warps, 64 rows each: per slab of 256 columns the nine 16-byte pieces that hold a
      // row's 128 bytes, wherever they start (the converters shift).
      role = 66;
      Ring raw;
      while (ok && walk.next(w)) {
        const int o0 = w.tile / p.r_tiles * kRows + (warp == 3 ? 64 : 0);
        const int end = min(w.s1 * kSlabK, p.columns);
        for (int column = w.s0 * kSlabK; column < end; column += kRawCols) {
          ok = mbar_wait_warp(&bars->raw_empty[raw.slot], raw.phase ^ 1u, abort_flag);
          if (!ok) break;
          uint8_t* dst = raw_ring + raw.slot * kRaw + (warp == 3 ? 64 : 0) * kLoosePitch;
#pragma unroll 6
          for (int i = 0; i < 64 * 9 / 32; ++i) {
            const int piece = i * 32 + lane;
            const int r = piece / 9;
            const long long from = ((static_cast<long long>(o0 + r) * p.row_bytes + column / 2) & ~15ll) +
                                   (piece - r * 9) * 16;
            // (bytes past the end of the codes, rows past the last: zeros, nothing is read)
            long long left = o0 + r < p.rows ? p.code_bytes - from : 0;
            const int size = left <= 0 ? 0 : (left > 16 ? 16 : static_cast<int>(left));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + piece * 16)),
                         "l"(p.panel + (size > 0 ? from : 0)), "r"(size)
                         : "memory");
          }
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bars->raw_full[raw.slot]))
                       : "memory");
          raw.advance(S::kRawSlots);
        }
      }
    } else if (warp == 0 && lane == 0) {
      // ------------------------------ packed codes ------------------------------
      role = 61;
      Ring raw;
      while (ok && walk.next(w)) {
        const int o_tile = w.tile / p.r_tiles;
        const int end = min(w.s1 * kSlabK, p.columns);
        for (int column = w.s0 * kSlabK; column < end; column += kRawCols) {
          ok = mbar_wait(&bars->raw_empty[raw.slot], raw.phase ^ 1u, abort_flag);
          if (!ok) break;
          uint8_t* dst = raw_ring + raw.slot * kRawBytes;
          mbar_arrive_expect_tx(&bars->raw_full[raw.slot], kRawBytes);
          if (SRC == kScaledPanelQ8) {
            const long long span = static_cast<long long>(o_tile) * p.slabs + column / kSlabK;
            const uint8_t* src = p.panel + span * slab_span_bytes(QX_FORMAT_Q8_0) +
                                 (column % kSlabK) / kRawCols * kRawBytes;
            bulk_load(dst, src, kRawBytes, &bars->raw_full[raw.slot]);
          } else {
            tma_load_2d(dst, &map_w, &bars->raw_full[raw.slot], column / kRawCols * 128, o_tile * kRows);
          }
          raw.advance(S::kRawSlots);
        }
      }
    } else if (warp == 2 && lane == 0) {
      // ------------------------------ activations -------------------------------
      role = 62;
      wait_for_kernel_in_front();
      Ring st;
      while (ok && walk.next(w)) {
        const int r0 = w.tile % p.r_tiles * p.bn;
        const int end = min(w.s1 * kSlabK, p.columns);
        for (int column = w.s0 * kSlabK; column < end; column += kStepCols) {
          ok = mbar_wait(&bars->empty[st.slot], st.phase ^ 1u, abort_flag);
          if (!ok) break;
          uint8_t* dst = smem + st.slot * stage_size + kStageA;
          mbar_arrive_expect_tx(&bars->full[st.slot], b_bytes);
          // (a sub-tile past the last column lies outside the tensor map's rows: zeros)
#pragma unroll
          for (int sub = 0; sub < kSubs; ++sub) {
#pragma unroll
            for (int plane = 0; plane < PLANES; ++plane) {
              tma_load_2d(dst + (sub * PLANES + plane) * b_sub, &map_x, &bars->full[st.slot],
                          column + sub * kSub, r0 + plane * p.m);
            }
          }
          st.advance(p.stages);
        }
      }
    } else if (warp == 1 && elect_one()) {
      // ------------------------------ MMA issuer --------------------------------
      role = 63;
      const uint32_t type = BF16 ? 1u : 0u;
      const uint32_t idesc = (1u << 4) | (type << 7) | (type << 10) |
                             (static_cast<uint32_t>(p.bn >> 3) << 17) |
                             (static_cast<uint32_t>(kRows >> 4) << 24);
      const uint64_t desc0 = make_sw128_kmajor_desc(smem_u32(smem));
      const uint32_t stage_units = stage_size >> 4, b_units = b_sub >> 4;
      const uint32_t hand_mask = static_cast<uint32_t>(p.hand_cols) - 1u;
      const uint32_t promote_mask = static_cast<uint32_t>(p.promote) - 1u;
      const int promote_log = p.promote_log, bn = p.bn;
      const uint32_t hand_size = static_cast<uint32_t>(bn) << (31 - __clz(p.hand_cols) - promote_log);
      Ring st, acc;
      while (ok && walk.next(w)) {
        const int end = min(w.s1 * kSlabK, p.columns);
        for (int column = w.s0 * kSlabK; column < end && ok; column += kStepCols) {
          ok = mbar_wait(&bars->full[st.slot], st.phase, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t a_desc = desc0 + st.slot * stage_units;
          const uint64_t b_desc = a_desc + (kStageA >> 4);
#pragma unroll
          for (int h = 0; h < 2 * kSubs; ++h) {  // 32 columns
            const uint32_t at = (column + 32 * h) & hand_mask;
            if (at == 0) {
              ok = mbar_wait(&bars->tmem_empty[acc.slot], acc.phase ^ 1u, abort_flag);
              if (!ok) break;
              tc_fence_after_sync();
            }
            const uint32_t d = tmem_base + acc.slot * hand_size + (at >> promote_log) * bn;
            uint32_t started = (at & promote_mask) != 0 ? 1u : 0u;
#pragma unroll
            for (int plane = PLANES - 1; plane >= 0; --plane) {  // (the small parts first)
              // 16 columns = 32 bytes inside the swizzle atom: +2 in the (address >> 4) field
              const uint64_t ad = a_desc + (h >> 1) * (kABytes >> 4) + 4 * (h & 1);
              const uint64_t bd = b_desc + ((h >> 1) * PLANES + plane) * b_units + 4 * (h & 1);
              mma_f16_ss(d, ad, bd, idesc, started);
              mma_f16_ss(d, ad + 2, bd + 2, idesc, 1u);
              started = 1u;
            }
            if (at + 32 == static_cast<uint32_t>(p.hand_cols)) {
              tc_commit(&bars->tmem_full[acc.slot]);
              acc.advance(p.accs);
            }
          }
          if (!ok) break;
          tc_commit(&bars->empty[st.slot]);
          st.advance(p.stages);
        }
      }
    }
  } else if (warp < 4 + S::kEpi) {
    // -------------------------------- epilogue ----------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::kEpiRegs));
    role = 64;
    wait_for_kernel_in_front();
    const int quarter = warp & 3;
    const int half = (warp - 4) >> 2;
    const int cols = p.bn / (S::kEpi / 4);  // columns of this warp
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                               static_cast<uint32_t>(half * cols);
    const uint32_t total_base = lane_base + static_cast<uint32_t>(kTmemCols - 2 * p.bn);
    const uint32_t hand_size = static_cast<uint32_t>(p.bn) << (31 - __clz(p.hand_cols) - p.promote_log);
    float* my_finish = finish + (warp - 4) * 32 * kFinishCols + lane;
    Ring acc;
    while (ok && walk.next(w)) {
      const int o_tile = w.tile / p.r_tiles;
      const int row = o_tile * kRows + quarter * 32 + lane;
      const bool live = row < p.rows;
      unsigned long long sum[S::kCols / 2];
#pragma unroll
      for (int i = 0; i < S::kCols / 2; ++i) sum[i] = 0ull;
      // Two levels of sums: chains of multiply-adds in registers, then each chain into a total and
      // what the total's roundings lost, both in TMEM columns behind the accumulators. So a result
      // is one chain's few roundings away from exact whatever the length of the row, and no
      // further than the separate lanes of the digit kernels leave it (q8_0, 11008 columns: 8.4e-8
      // of the result, digit kernels 9.6e-8, one chain over all units 2.4e-7; 1024 columns: 6.2e-8
      // and 6.6e-8). Whole numbers (W4A8) are exact in one chain. Not in registers or local
      // memory: the former are full, the latter has next to no L1 beside the shared memory.
      // A total costs 4 % of 512 tokens on 14336 x 4096 uint4, 11 % of 331 on 4096 x 11008 q8_0.
      bool flushed = false;
      auto flush = [&]() {
        if (flushed) tmem_st_wait();
#pragma unroll
        for (int c = 0; c < S::kCols; c += 8) {  // (few columns at a time: the registers are full)
          if (c >= cols) break;
          uint32_t total[8], rest[8];
          if (flushed) {
            tmem_ld_32x8(total_base + c, total);
            tmem_ld_32x8(total_base + p.bn + c, rest);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) total[i] = rest[i] = 0u;
          }
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            unsigned long long t = pack2(total[i], total[i + 1]), r = pack2(rest[i], rest[i + 1]);
            add_with_rest2(t, r, sum[(c + i) / 2]);
            sum[(c + i) / 2] = 0ull;
            unpack2(t, total[i], total[i + 1]);
            unpack2(r, rest[i], rest[i + 1]);
          }
          tmem_st_32x8(total_base + c, total);
          tmem_st_32x8(total_base + p.bn + c, rest);
        }
        flushed = true;
      };
      // Waits for the accumulators of the next hand-over; false when the kernel gives up.
      auto take = [&]() {
        ok = mbar_wait_warp(&bars->tmem_full[acc.slot], acc.phase, abort_flag);
        tc_fence_after_sync();
        return ok;
      };
      // sum += scale * accumulators at `taddr`; `release`: the last ones of the hand-over.
      // 16 columns at a time: with 32 of them in registers the loop spills (q8_0, 331 tokens on
      // 4096 x 11008: 147 us against 139).
      auto add_unit = [&](uint32_t taddr, float scale, bool release) {
        if (BF16) scale *= kBf16Unscale;
        const unsigned long long s2 = pack2(__float_as_uint(scale), __float_as_uint(scale));
#pragma unroll
        for (int c = 0; c < S::kCols; c += 16) {
          if (c >= cols) break;
          uint32_t v[16];
          tmem_ld_32x16(taddr + c, v);
          tmem_ld_wait();
          if (release && c + 16 >= cols) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->tmem_empty[acc.slot]);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) fma2(sum[c / 2 + j], pack2(v[2 * j], v[2 * j + 1]), s2);
        }
      };
      const float* row_scales = p.scales + static_cast<long long>(live ? row : 0) * p.groups;
      if (SRC == kScaledPanelQ8) {
        // scales come one slab (eight units) ahead; a chain is one slab, or two
        const int hand_units = S::kEpi == 16 ? 1 : p.hand_cols / 32;
        int pending = 0;
        const uint8_t* slab_scales = p.panel + (static_cast<long long>(o_tile) * p.slabs + w.s0) * slab_span_bytes(QX_FORMAT_Q8_0) +
                                     panel_scale_offset(QX_FORMAT_Q8_0, quarter * 32 + lane, 0);
        uint4 next = __ldg(reinterpret_cast<const uint4*>(slab_scales));
        for (int s = w.s0; s < w.s1 && ok; ++s) {
          uint4 blocks = next;
          slab_scales += slab_span_bytes(QX_FORMAT_Q8_0);
          if (s + 1 < w.s1) next = __ldg(reinterpret_cast<const uint4*>(slab_scales));
          const int units = min(kSlabK, p.columns - s * kSlabK) / 32;
          for (int u = 0; u < units; ++u) {
            const int at = u & (hand_units - 1);
            if (at == 0 && !take()) break;
            const bool last = at == hand_units - 1;
            add_unit(lane_base + acc.slot * hand_size + at * p.bn,
                     half_bits_to_float(static_cast<unsigned short>(blocks.x)), last);
            if (last) acc.advance(p.accs);
            blocks.x = __funnelshift_r(blocks.x, blocks.y, 16);
            blocks.y = __funnelshift_r(blocks.y, blocks.z, 16);
            blocks.z = __funnelshift_r(blocks.z, blocks.w, 16);
            blocks.w >>= 16;
          }
          pending += kSlabK / 32;
          if (pending == p.chain && s + 1 < w.s1) {
            pending = 0;
            flush();
          }
        }
      } else {
        const int begin = w.s0 * kSlabK;
        const int end = min(w.s1 * kSlabK, p.columns);
        const int hand_units = p.hand_cols >> p.promote_log;
        int pending = 0;
        // scale of the unit at `column`, fetched one group ahead
        int g = begin / p.group;
        int boundary = (g + 1) * p.group;
        float scale = 1.0f, next_scale = 1.0f;
        if (p.token_scales == nullptr) {  // (whole numbers are summed; the scales come at the end)
          scale = live ? __ldg(row_scales + g) : 0.0f;
          next_scale = live && g + 1 < p.groups ? __ldg(row_scales + g + 1) : 0.0f;
        }
        for (int column = begin; column < end; column += p.hand_cols) {
          if (!take()) break;
          uint32_t taddr = lane_base + acc.slot * hand_size;
          const int hand_end = min(column + p.hand_cols, end);
          for (int unit = column; unit < hand_end; unit += p.promote, taddr += p.bn) {
            if (unit >= boundary) {
              scale = next_scale;  // (0 past the last group: padding columns of the last stage)
              ++g;
              boundary += p.group;
              next_scale = live && g + 1 < p.groups ? __ldg(row_scales + g + 1) : 0.0f;
            }
            add_unit(taddr, scale, unit + p.promote >= hand_end);
          }
          acc.advance(p.accs);
          pending += hand_units;  // (1, 2 or 4)
          if (pending == p.chain && column + p.hand_cols < end && p.token_scales == nullptr) {
            pending = 0;
            flush();
          }
        }
      }
      if (!ok) break;
      flush();
      tmem_st_wait();
      // Finish the tile, kFinishCols columns at a time in ROLLED loops: this code runs once per
      // tile, and unrolled it costs more in instruction fetches than in work. A piece of a tile
      // goes to scratch; whoever completes the tile's count adds the pieces in CTA order.
      auto finished = [&](int c, float (&out)[kFinishCols]) {
        uint32_t total[kFinishCols], rest[kFinishCols];
        tmem_ld_32x16(total_base + c, total);
        tmem_ld_32x16(total_base + p.bn + c, rest);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < kFinishCols; ++i) {  // (a total that is not finite has no rest)
          const float t = __uint_as_float(total[i]);
          out[i] = isfinite(t) ? t + __uint_as_float(rest[i]) : t;
        }
      };
      const size_t slot_floats = static_cast<size_t>(kRows) * p.bn;
      const size_t mine = static_cast<size_t>(half * cols) * kRows + quarter * 32 + lane;
      const bool piece = p.split && !(w.s0 == 0 && w.s1 == p.slabs);
      const int token0 = w.tile % p.r_tiles * p.bn + half * cols;
      const int tokens = min(p.m - token0, cols);  // may be < 1
      const long long u0 = static_cast<long long>(w.tile) * p.slabs;
      int c0 = 0, c1 = 0;  // CTAs that hold pieces of the tile
      if (piece) {
        c0 = static_cast<int>(((u0 + 1) * gridDim.x - 1) / p.units);
        c1 = static_cast<int>(((u0 + p.slabs) * gridDim.x - 1) / p.units);
      }
      auto piece_of = [&](int c) {  // (a CTA's first tile has slot 0, its last one slot 1)
        const long long first = (p.units * c / gridDim.x) / p.slabs;
        return p.partial + (2 * static_cast<size_t>(c) + (first == w.tile ? 0 : 1)) * slot_floats + mine;
      };
      if (piece) {
        float* own = piece_of(blockIdx.x);
#pragma unroll 1
        for (int c = 0; c < tokens; c += kFinishCols) {
          float part[kFinishCols];
          finished(c, part);
#pragma unroll
          for (int i = 0; i < kFinishCols; ++i) __stcg(own + i * kRows, part[i]);
          own += kFinishCols * kRows;
        }
        __threadfence();
        __syncwarp();
        // (a CTA is the first of at most two tiles: the count lives beside its piece's slot)
        const int c0_first = static_cast<int>((p.units * c0 / gridDim.x) / p.slabs);
        int* counter = p.counters + (2 * c0 + (c0_first == w.tile ? 0 : 1)) * S::kEpi + (warp - 4);
        int before = 0;
        if (lane == 0) before = atomicAdd(counter, 1);
        before = __shfl_sync(0xffffffffu, before, 0);
        if (before != c1 - c0) continue;
        if (lane == 0) *counter = 0;
        __threadfence();
      }
      const float bias = p.bias != nullptr && live ? __ldg(p.bias + row) : 0.0f;
      const float row_scale = p.token_scales != nullptr && live ? __ldg(row_scales) : 1.0f;
      long long at = token0 * p.ldy + row;
#pragma unroll 1
      for (int c = 0; c < tokens; c += kFinishCols) {
        if (piece) {  // (in 64 bits: a piece adds no rounding but its own)
          double whole[kFinishCols];
#pragma unroll
          for (int i = 0; i < kFinishCols; ++i) whole[i] = 0.0;
#pragma unroll 2
          for (int k = c0; k <= c1; ++k) {
            const float* in = piece_of(k) + c * kRows;
#pragma unroll
            for (int i = 0; i < kFinishCols; ++i) whole[i] += __ldcg(in + i * kRows);
          }
#pragma unroll
          for (int i = 0; i < kFinishCols; ++i) my_finish[i * 32] = static_cast<float>(whole[i]);
        } else {
          float part[kFinishCols];
          finished(c, part);
#pragma unroll
          for (int i = 0; i < kFinishCols; ++i) my_finish[i * 32] = part[i];
        }
        const int count = tokens - c < kFinishCols ? tokens - c : kFinishCols;
        if (live) {
#pragma unroll 4
          for (int j = 0; j < count; ++j) {
            float out = my_finish[j * 32] + bias;
            if (p.token_scales != nullptr) {
              out = __fmul_rn(__fmul_rn(out, row_scale), __ldg(p.token_scales + token0 + c + j));
            } else if (p.activation != QX_ACTIVATION_NONE) {
              out = projection_activation(out, p.activation);
            }
            const long long where = at + j * p.ldy;
            if (p.y_type == QX_STORAGE_F32) {
              static_cast<float*>(p.y)[where] = out;
            } else {
              static_cast<uint16_t*>(p.y)[where] =
                  p.y_type == QX_STORAGE_F16 ? __half_as_ushort(__float2half_rn(out)) : storage_bf16_bits(out);
            }
          }
          at += kFinishCols * p.ldy;
        }
      }
    }
    tmem_st_wait();  // (of totals, where the kernel gave up in the middle of a tile)
  } else {
    // -------------------------------- converters --------------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::kConvRegs));
    role = 65;
    // A thread converts one sub-tile (64 columns) of its row per stage. A group of eight warps
    // takes every stage, or two groups take them in turn, strictly, across the ends of tiles as
    // well: a parity wait is sound only where the phase before it is known to be over. A group
    // that left out two stages in a row (an odd number of them in a tile, and the next tile's
    // first one given to the same group again) would take the stage of two rounds ago for free.
    const int cw = warp - 4 - S::kEpi;
    const int r = (cw & 3) * 32 + lane;
    const int sub = (cw >> 2) & 1, group = cw >> 3;
    const int swizzle = r & 7;
    int turn = 0;  // the group whose stage it is
    Ring raw, st;
    while (ok && walk.next(w)) {
      const int row = w.tile / p.r_tiles * kRows + r;
      const int end = min(w.s1 * kSlabK, p.columns);
      // zero points, one 32-column half ahead
      const int first_byte = static_cast<int>((static_cast<long long>(row) * p.row_bytes) & 15);
      const bool zeros = kNibbles && p.zeros != nullptr;
      const float* row_zeros = zeros ? p.zeros + static_cast<long long>(row < p.rows ? row : 0) * p.groups : nullptr;
      int g = 0;
      int boundary = 0x7fffffff;
      float next_zero = 8.0f;
      bool fetched = false;
      uint32_t base_z = zero_word<BF16>(8.0f);
      if (zeros) {
        const int column = w.s0 * kSlabK + sub * kSub + (S::kGroups == 2 && turn != group ? kStepCols : 0);
        g = column / p.group;
        boundary = (g + 1) * p.group;
        next_zero = g < p.groups ? __ldg(row_zeros + g) : 0.0f;
        fetched = true;
      }
      for (int column = w.s0 * kSlabK; column < end; column += kStepCols) {
        const int in_slot = column % kRawCols;
        const bool release = in_slot + kStepCols == kRawCols || column + kStepCols >= end;
        const bool mine = S::kGroups == 1 || turn == group;
        turn ^= 1;
        if (!mine) {
          // the other group's stage; a last slot of nibbles with that stage alone is given back
          // by both groups
          if (kNibbles && release && in_slot == 0) {
            ok = mbar_wait_warp(&bars->raw_full[raw.slot], raw.phase, abort_flag);
            if (!ok) break;
            if (lane == 0) mbar_arrive(&bars->raw_empty[raw.slot]);
          }
          st.advance(p.stages);
          if (release) raw.advance(S::kRawSlots);
          continue;
        }
        // (the stage first: its last but one use is over, as this group has waited for that or for
        // a later one, and that it is free says the same of the slots of packed codes)
        ok = mbar_wait_warp(&bars->empty[st.slot], st.phase ^ 1u, abort_flag);
        if (!ok) break;
        if (in_slot == 0 || S::kGroups == 2) {
          ok = mbar_wait_warp(&bars->raw_full[raw.slot], raw.phase, abort_flag);
          if (!ok) break;
        }
        const uint8_t* src = raw_ring + raw.slot * kRaw + r * (kLoose ? kLoosePitch : 128);
        uint8_t* stage = smem + st.slot * stage_size + r * 128;
        {
          uint8_t* dst = stage + sub * kABytes;
          const int at = column + sub * kSub;             // first column of the sub-tile
          const int half = (in_slot + sub * kSub) / 32;   // 32-column halves inside the slot
          if (kNibbles) {
            uint4 packed[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (kLoose) {
                const int byte = first_byte + (half + h) * 16;
                const uint32_t* word = reinterpret_cast<const uint32_t*>(src) + (byte >> 2);
                const uint32_t shift = (byte & 3) * 8;
                uint32_t x[5];
#pragma unroll
                for (int q = 0; q < 5; ++q) x[q] = word[q];
                packed[h] = make_uint4(__funnelshift_r(x[0], x[1], shift), __funnelshift_r(x[1], x[2], shift),
                                       __funnelshift_r(x[2], x[3], shift), __funnelshift_r(x[3], x[4], shift));
              } else {
                packed[h] = *reinterpret_cast<const uint4*>(src + (((half + h) ^ swizzle) << 4));
              }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (fetched) {
                // (the pin keeps the conversion here: right behind its load it would wait for it)
                asm volatile("" : "+f"(next_zero));
                base_z = zero_word<BF16>(next_zero);
                fetched = false;
              }
              // the zero point of the thread's next half, if its group is another one
              const int next_column = at + (h == 0 ? 32 : kStepCols * S::kGroups);
              if (next_column >= boundary) {
                do {
                  ++g;
                  boundary += p.group;
                } while (next_column >= boundary);
                next_zero = g < p.groups ? __ldg(row_zeros + g) : 0.0f;
                fetched = true;
              }
              const uint4 v = packed[h];
              const uint32_t words[4] = {v.x ^ p.nibble_xor, v.y ^ p.nibble_xor, v.z ^ p.nibble_xor,
                                         v.w ^ p.nibble_xor};
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                *reinterpret_cast<uint4*>(dst + (((4 * h + q) ^ swizzle) << 4)) =
                    convert_nibbles<BF16>(words[q], base_z);
              }
            }
          } else {
            uint4 packed[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              packed[q] = *reinterpret_cast<const uint4*>(src + (((2 * half + q) ^ swizzle) << 4));
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint4 v = packed[q];
              *reinterpret_cast<uint4*>(dst + (((2 * q) ^ swizzle) << 4)) =
                  make_uint4(convert_bytes2<BF16>(v.x, 0x4140u), convert_bytes2<BF16>(v.x, 0x4342u),
                             convert_bytes2<BF16>(v.y, 0x4140u), convert_bytes2<BF16>(v.y, 0x4342u));
              *reinterpret_cast<uint4*>(dst + (((2 * q + 1) ^ swizzle) << 4)) =
                  make_uint4(convert_bytes2<BF16>(v.z, 0x4140u), convert_bytes2<BF16>(v.z, 0x4342u),
                             convert_bytes2<BF16>(v.w, 0x4140u), convert_bytes2<BF16>(v.w, 0x4342u));
            }
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bars->full[st.slot]);
          // (all lanes have read before the __syncwarp)
          if (release || (S::kGroups == 2 && kNibbles)) mbar_arrive(&bars->raw_empty[raw.slot]);
        }
        st.advance(p.stages);
        if (release) raw.advance(S::kRawSlots);
      }
    }
  }
  if (!ok) {
    *abort_flag = 1;
    report_error(p.error, role);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Activations that the kernel cannot read in place: f32 (three bf16 planes [plane][m][columns],
// each the truncated remainder of the ones before, so that their sum is the value), act-order
// tensors (gathered into packed order), and 16-bit rows that do not start on 16 bytes.
__global__ void __launch_bounds__(256) stage_activations_kernel(const void* __restrict__ x, int x_type,
                                                                const int* __restrict__ order,
                                                                uint16_t* __restrict__ out,
                                                                long long columns, long long m) {
  asm volatile("griddepcontrol.launch_dependents;");
  wait_for_kernel_in_front();
  const long long total = m * columns;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    long long from = i;
    if (order != nullptr) {
      const long long token = i / columns;
      from = token * columns + order[i - token * columns];
    }
    if (x_type == QX_STORAGE_F32) {
      const float v = static_cast<const float*>(x)[from];
      const uint32_t hi = __float_as_uint(v) & 0xffff0000u;
      const float r1 = v - __uint_as_float(hi);
      const uint32_t mid = __float_as_uint(r1) & 0xffff0000u;
      const float r2 = r1 - __uint_as_float(mid);
      out[i] = static_cast<uint16_t>(hi >> 16);
      out[total + i] = static_cast<uint16_t>(mid >> 16);
      out[2 * total + i] = static_cast<uint16_t>(__float_as_uint(r2) >> 16);
    } else {
      out[i] = static_cast<const uint16_t*>(x)[from];
    }
  }
}

struct Plan {
  bool small, staged, split;
  int bn, planes, promote, slabs, columns, o_tiles, r_tiles, grid;
  size_t staged_bytes;
};

Plan make_plan(const ScaledGemmArgs& a, int sm_count) {
  Plan p{};
  p.planes = a.x_type == QX_STORAGE_F32 ? 3 : 1;
  p.staged = p.planes == 3 || a.order != nullptr || reinterpret_cast<uintptr_t>(a.x) % 16 != 0;
  p.staged_bytes = p.staged ? align_up(static_cast<size_t>(p.planes) * a.m * a.columns * 2, 256) : 0;
  p.promote = a.group % 128 == 0 || a.group == a.columns ? 128 : (a.group % 64 == 0 ? 64 : 32);
  // Three planes: the sums of 64 columns leave the tensor core, or its own f32 adds would show
  // (scale groups of 128: 3.2e-7 of the result after 128 columns each, 1.5e-7 after 64, digit
  // kernels 2.3e-7 to 2.5e-7; bytes 3.5e-7 and 1.7e-7). And f16 activations on bytes, products of
  // 18 bits, those of 32 columns (groups of 128: 1.2e-7 after 128 columns, 7.5e-8 after 32, digit
  // kernels 7.0e-8 to 9.8e-8).
  if (p.planes == 3 && p.promote > 64) p.promote = 64;
  if (a.source == kScaledBytes && a.x_type == QX_STORAGE_F16) p.promote = 32;
  p.small = a.m <= Small::kTokens || p.planes == 3;  // (three planes of 128 tokens: no two stages)
  const int most = p.small ? Small::kTokens : Large::kTokens;
  p.r_tiles = static_cast<int>((a.m + most - 1) / most);
  // (an epilogue warp takes half of a tile's tokens, 32 at a time; one tile of up to 32 tokens
  // leaves its second half idle)
  const int unit = 64;
  p.bn = a.m <= 32 ? 32 : static_cast<int>(((a.m + p.r_tiles - 1) / p.r_tiles + unit - 1) / unit * unit);
  p.slabs = static_cast<int>((a.columns + kSlabK - 1) / kSlabK);
  p.columns = static_cast<int>((a.columns + kStepCols - 1) / kStepCols * kStepCols);
  p.o_tiles = static_cast<int>((a.rows + kRows - 1) / kRows);
  const long long tiles = static_cast<long long>(p.o_tiles) * p.r_tiles;
  const long long units = tiles * p.slabs;
  // Whole tiles, or equal ranges of slabs? The slowest CTA has ceil(tiles / SMs) whole tiles or
  // ceil(units / SMs) slabs and the cost of handing pieces on, about two slabs.
  const long long whole = (tiles + sm_count - 1) / sm_count * p.slabs;
  const long long even = (units + sm_count - 1) / sm_count + 2;
  p.split = !a.whole_tiles && even < whole && units < (1LL << 30);
  const long long pieces = p.split ? units : tiles;
  p.grid = static_cast<int>(pieces < sm_count ? pieces : sm_count);
  return p;
}

template <int SRC, bool BF16, int PLANES, class S>
qx_status launch_kernel(const CUtensorMap& map_w, const CUtensorMap& map_x, ScaledParams& p, int grid,
                        cudaStream_t stream) {
  p.stages = stages_for<S>(p.bn, PLANES, raw_bytes(SRC));
  p.promote_log = p.promote == 128 ? 7 : (p.promote == 64 ? 6 : 5);
  // one hand-over of accumulators per stage, or shorter ones where two would not fit beside the
  // totals and their rests
  const int free_cols = kTmemCols - 2 * p.bn;
  p.hand_cols = kStepCols;
  while (p.hand_cols > p.promote && 2 * p.bn * (p.hand_cols / p.promote) > free_cols) p.hand_cols /= 2;
  const int hand = p.bn * (p.hand_cols / p.promote);
  p.accs = free_cols / hand > kMaxAcc ? kMaxAcc : free_cols / hand;
  p.chain = p.columns >> p.promote_log >= kLongRowUnits ? kLongChain : kChain;
  if (p.accs < 2 || (SRC == kScaledPanelQ8 && S::kEpi == 16 && p.hand_cols != 32)) {
    set_last_error_text("scaled projection: accumulators beyond TMEM");
    return QX_STATUS_DEVICE_ERROR;
  }
  static SmemOptIn opt_in;
  QX_TRY(opt_in.ensure(scaled_gemm_kernel<SRC, BF16, PLANES, S>, kSmemMax));
  // the warpgroups' register shares have to fit what the block is launched with
  static const int registers = [] {
    cudaFuncAttributes attributes{};
    return cudaFuncGetAttributes(&attributes, scaled_gemm_kernel<SRC, BF16, PLANES, S>) == cudaSuccess
               ? attributes.numRegs
               : 0;
  }();
  if (registers / 8 * 8 * (S::kThreads / 128) < S::kRegShares) {
    set_last_error_text("scaled projection: the kernel was compiled with too few registers");
    return QX_STATUS_DEVICE_ERROR;
  }
  cudaLaunchAttribute attribute{};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(static_cast<unsigned>(grid));
  config.blockDim = dim3(S::kThreads);
  config.dynamicSmemBytes = other_bytes<S>(raw_bytes(SRC)) + p.stages * stage_bytes<S>(p.bn, PLANES);
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = 1;
  QX_CUDA_TRY(cudaLaunchKernelEx(&config, scaled_gemm_kernel<SRC, BF16, PLANES, S>, map_w, map_x,
                                 static_cast<const ScaledParams&>(p)));
  count_launch();
  return QX_STATUS_OK;
}
template <int SRC>
qx_status launch_source(bool small, int x_type, const CUtensorMap& map_w, const CUtensorMap& map_x,
                        ScaledParams& p, int grid, cudaStream_t stream) {
  if (x_type == QX_STORAGE_F32) {
    return launch_kernel<SRC, true, 3, SmallPlanes>(map_w, map_x, p, grid, stream);
  }
  if (x_type == QX_STORAGE_F16) {
    return small ? launch_kernel<SRC, false, 1, Small>(map_w, map_x, p, grid, stream)
                 : launch_kernel<SRC, false, 1, Large>(map_w, map_x, p, grid, stream);
  }
  return small ? launch_kernel<SRC, true, 1, Small>(map_w, map_x, p, grid, stream)
               : launch_kernel<SRC, true, 1, Large>(map_w, map_x, p, grid, stream);
}

}  // namespace

bool scaled_gemm_serves(const ScaledGemmArgs& a) {
  if (a.source == kScaledPanelQ8 && a.x_type != QX_STORAGE_BF16) return false;
  if (a.m < 1 || a.m > 65535 || a.rows < 1 || a.rows > (1LL << 26) || a.columns > (1LL << 24)) return false;
  // rows of codes and of activations start on 16 bytes, groups on a converter's 32 columns
  if (a.source == kScaledNibblesLoose) {  // (activations in rows of whole 16-byte vectors)
    return a.m > Small::kTokens && a.group == a.columns && a.token_scales != nullptr && a.x_type == QX_STORAGE_F16 &&
           a.x_stride % 8 == 0 && reinterpret_cast<uintptr_t>(a.codes) % 16 == 0;
  }
  const long long row_bytes = a.source == kScaledNibbles ? a.columns / 2 : a.columns;
  if (a.source == kScaledNibbles && a.columns % 2 != 0) return false;
  if (row_bytes % 16 != 0 || a.columns % 8 != 0 || reinterpret_cast<uintptr_t>(a.codes) % 16 != 0) return false;
  return a.group == a.columns || a.group % 32 == 0;
}

size_t scaled_gemm_scratch_bytes(const ScaledGemmArgs& a, int sm_count) {
  const int planes = a.source == kScaledPanelQ8 ? 1 : 3;
  const size_t tokens = a.m <= 32 ? 32 : (a.m <= 64 ? 64 : Large::kTokens);
  return align_up(static_cast<size_t>(planes) * a.m * a.columns * 2, 256) +
         static_cast<size_t>(sm_count) * 2 * kRows * tokens * sizeof(float);
}

qx_status launch_scaled_gemm(const ScaledGemmArgs& a, void* scratch, int* counters, size_t counter_bytes,
                             int sm_count, int* error, cudaStream_t stream) {
  const Plan plan = make_plan(a, sm_count);
  if (plan.split && scaled_gemm_counter_bytes(plan.grid) > counter_bytes) {
    set_last_error_text("scaled projection: more pieces than arrival counters");
    return QX_STATUS_DEVICE_ERROR;
  }
  const void* x = a.x;
  if (plan.staged) {
    const long long blocks = (a.m * a.columns + 255) / 256;
    const long long cap = 8LL * sm_count;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(blocks < cap ? blocks : cap));
    config.blockDim = dim3(256);
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    QX_CUDA_TRY(cudaLaunchKernelEx(&config, stage_activations_kernel, a.x, a.x_type, a.order,
                                   static_cast<uint16_t*>(scratch), a.columns, a.m));
    count_launch();
    x = scratch;
  }
  const bool bf16 = a.x_type != QX_STORAGE_F16;
  CUtensorMap map_x{}, map_w{};
  bool encoded = encode_tma_2d(&map_x, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                               x, static_cast<uint64_t>(a.columns), static_cast<uint64_t>(plan.planes * a.m),
                               static_cast<uint64_t>(a.x_stride != 0 && !plan.staged ? a.x_stride : a.columns) * 2, kSub, static_cast<uint32_t>(plan.bn));
  if (a.source != kScaledPanelQ8 && a.source != kScaledNibblesLoose) {
    const uint64_t row_bytes = static_cast<uint64_t>(a.source == kScaledNibbles ? a.columns / 2 : a.columns);
    encoded = encoded && encode_tma_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.codes, row_bytes,
                                       static_cast<uint64_t>(a.rows), row_bytes, 128, kRows);
  }
  if (!encoded) {
    set_last_error_text("cuTensorMapEncodeTiled failed for a scaled projection");
    return QX_STATUS_DEVICE_ERROR;
  }
  ScaledParams p{};
  p.panel = a.codes;
  p.scales = a.scales;
  p.zeros = a.zeros;
  p.bias = a.bias;
  p.token_scales = a.token_scales;
  p.row_bytes = (a.columns + 1) / 2;
  p.code_bytes = p.row_bytes * a.rows;
  p.y = a.y;
  p.partial = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + plan.staged_bytes);
  p.counters = counters;
  p.error = error;
  p.m = static_cast<int>(a.m);
  p.rows = static_cast<int>(a.rows);
  p.ldy = a.ldy;
  p.group = static_cast<int>(a.group);
  p.groups = a.group == a.columns ? 1 : static_cast<int>(a.columns / a.group);
  p.units = static_cast<long long>(plan.o_tiles) * plan.r_tiles * plan.slabs;
  p.nibble_xor = a.nibble_xor;
  p.columns = plan.columns;
  p.slabs = plan.slabs;
  p.bn = plan.bn;
  p.promote = plan.promote;
  p.o_tiles = plan.o_tiles;
  p.r_tiles = plan.r_tiles;
  p.split = plan.split ? 1 : 0;
  p.y_type = a.y_type;
  p.activation = a.activation;
  const bool small = plan.small;
  switch (a.source) {
    case kScaledNibbles:
      return launch_source<kScaledNibbles>(small, a.x_type, map_w, map_x, p, plan.grid, stream);
    case kScaledNibblesLoose:  // (f16 activations, more tokens than a small tile has)
      return launch_kernel<kScaledNibblesLoose, false, 1, Large>(map_w, map_x, p, plan.grid, stream);
    case kScaledBytes:
      return launch_source<kScaledBytes>(small, a.x_type, map_w, map_x, p, plan.grid, stream);
    default:  // (bf16 activations only)
      return small ? launch_kernel<kScaledPanelQ8, true, 1, Small>(map_w, map_x, p, plan.grid, stream)
                   : launch_kernel<kScaledPanelQ8, true, 1, Large>(map_w, map_x, p, plan.grid, stream);
  }
}

}  // namespace qx
