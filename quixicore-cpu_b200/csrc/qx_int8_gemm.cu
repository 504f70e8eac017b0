// W8A8 dispatch: picks the tensor-core kernel when the operands meet its alignment rules,
// otherwise the any-shape CUDA-core kernel. Mirrors the variant table of the reference
// (src/dispatch/int8_gemm.cpp:20-63): the choice is resolved once per process and
// QX_B200_INT8_GEMM_VARIANT=dp4a forces the CUDA-core kernel for A/B checks, as
// QUIXICORE_CPU_INT8_GEMM_VARIANT does there. Both are GPU kernels; there is no CPU path.

#include <cstdlib>
#include <cstring>

#include "qx_int8_gemm.cuh"
#include "qx_stream_mma.cuh"

namespace qx {

bool int8_gemm_forced_simple() {
  static const bool forced = []() {
    const char* v = std::getenv("QX_B200_INT8_GEMM_VARIANT");
    return v != nullptr && std::strcmp(v, "dp4a") == 0;
  }();
  return forced;
}

const char* int8_gemm_variant_name() {
  return int8_gemm_forced_simple() ? "sm100a_dp4a" : "sm100a_tcgen05_i8";
}

namespace {
// Batches that qx_stream_mma.cu takes: few rows, where a tile of 128 or 256 channels leaves most SMs idle
// (us, there | tensor-core kernel): 1024 x 1408, 4 rows 2.9 | 6.2;  4096 x 4096: 1: 5.5 | 8.7, 16: 6.2 | 9.2,
// 24: 7.6 | 9.4;  8192 x 4096: 16: 8.0 | 14.3, 24: 11.3 | 14.9;  14336 x 4096: 4: 14.9 | 16.5, 16: 16.9 | 17.1,
// 32: 23 | 15.4;  4096 x 8192: 32: 13.5 | 23.6;  4096 x 4096: 64: 10.6 | 9.0.
bool stream_route(const Int8GemmArgs& a, StreamIntArgs* s) {
  if (a.m > 32 || (a.m > 8 && a.m * a.n > (1LL << 18))) return false;
  s->source = kStreamBytes;
  s->result = kStreamW8A8;
  s->codes = reinterpret_cast<const uint8_t*>(a.w);
  s->x = a.x;
  s->x_rows = static_cast<int>(a.m);
  s->rows = a.n;
  s->columns = a.k;
  s->ws = a.ws;
  s->as = a.as;
  s->row_sum = a.asymmetric ? a.row_sum : nullptr;
  s->zp = a.zp;
  s->y = a.y;
  s->y_type = QX_STORAGE_F32;
  s->ldy = a.ldy;
  s->acc = a.acc;
  return stream_int_serves(*s);
}
}  // namespace

qx_status launch_int8_gemm(const Int8GemmArgs& a, cudaStream_t stream) {
  StreamIntArgs s{};
  if (!int8_gemm_forced_simple() && stream_route(a, &s)) return launch_stream_int(s, stream);
  if (!int8_gemm_forced_simple() && int8_gemm_tc_supported(a)) return launch_int8_gemm_tc(a, stream);
  return launch_int8_gemm_simple(a, stream);
}

}  // namespace qx
