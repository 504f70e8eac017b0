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
// Batches that qx_stream_mma.cu takes: few rows on few channels, where tiles of 128 channels leave most SMs idle. With more
// channels they do not, and the TMA rings of the tensor-core kernel read faster than the streamed loads; of longer rows the
// warps' loads spread over more of them. Measured in graph replay (us, there | tensor-core kernel):
//   1 row:   1024 x 1408 3.1 | 5.9;  4096 x 4096 7.5 | 9.8;  8192 x 4096 9.1 | 11.6;  4096 x 11008 15.4 | 18.3;
//     11008 x 4096 15.0 | 14.2;  14336 x 8192 27.7 | 25.3;  28672 x 8192 52.5 | 46.6;  8192 x 28672 49.6 | 48.1
//   16 rows: 4096 x 4096 7.6 | 10.2;  5120 x 5120 10.5 | 11.7;  8192 x 4096 10.2 | 11.9;  14336 x 4096 17.8 | 14.5;
//     8192 x 28672 52 | 49
//   24 rows: 4096 x 4096 8.8 | 10.4;  2048 x 8192 13.4 | 14.5;  4096 x 11008 18.5 | 18.9;  4096 x 28672 41.9 | 40.6;
//     5120 x 5120 15.2 | 11.7
//   32 rows, a whole tile of tokens there: 1024 x 1024 3.5 | 3.8;  2000 x 2048 5.4 | 5.5;  1000 x 4096 7.2 | 7.5;
//     3000 x 4096 8.5 | 7.9
bool few_rows(const Int8GemmArgs& a) {
  if (a.m == kStreamW8A8Rows) return a.n <= 4096 && a.n * a.k <= (1LL << 22);
  if (a.n <= 4096 && a.m < kStreamW8A8Rows) return a.m <= 16 || a.k <= 16384;
  return a.n <= 8192 && a.m <= 16 && a.k <= 16384;
}
bool stream_route(const Int8GemmArgs& a, StreamIntArgs* s) {
  if (!few_rows(a)) return false;
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
