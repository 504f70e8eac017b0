"""Both sides of the lines between the streamed small batches (csrc/qx_stream_mma.cu) and the routes beside them: W8A8 bit
for bit, canonical tensors against float64 within the reference test's own 4e-5 * (1 + |exact|)."""

import numpy as np
import pytest

from test_canonical_gpu import BF16, F16, F32, INT4, INT8, UINT4, close
from test_scaled_gemm_gpu import _product_f64, _storage, _tensor

pytestmark = pytest.mark.gpu


# 16 | 17 rows, 31 | 32 rows, 4096 | 4097 and 8192 | 8193 channels, 16384 | 16400 columns; one and two tiles of rows per warp
@pytest.mark.parametrize("m,n,k", [(1, 8193, 1024), (16, 8192, 1040), (16, 4736, 528), (16, 4737, 528), (17, 4096, 1040),
                                   (17, 4097, 272), (31, 4096, 272), (32, 4096, 272), (31, 700, 16384), (31, 700, 16400),
                                   (2, 4097, 16400), (9, 6143, 272)])
def test_w8a8(qx, m, n, k):
    rng = np.random.Generator(np.random.Philox(key=[m * 7 + n, k]))
    w, x = rng.integers(-128, 128, (n, k), dtype=np.int8), rng.integers(-128, 128, (m, k), dtype=np.int8)
    ws, xs = rng.uniform(0.001, 0.01, n).astype(np.float32), rng.uniform(0.005, 0.05, m).astype(np.float32)
    row_sum, zp = w.sum(axis=1, dtype=np.int32), rng.integers(-20, 21, m, dtype=np.int32)
    acc = x.astype(np.float64) @ w.astype(np.float64).T - zp.astype(np.float64)[:, None] * row_sum.astype(np.float64)[None, :]
    status, y = qx.int8_gemm(w, x, ws, xs, m, n, k, row_sum=row_sum, zp=zp, asymmetric=True)
    assert status == qx.OK, qx.last_error()
    assert np.array_equal(y.view(np.uint32), ((acc.astype(np.float32) * ws[None, :]) * xs[:, None]).view(np.uint32))


@pytest.mark.parametrize("layout,group,n,k,m,x_type", [
    (INT8, 0, 4737, 1072, 2, BF16),     # digits: two tiles of rows per warp below 6144 rows
    (INT8, 0, 8192, 528, 8, F16), (INT8, 0, 8193, 528, 8, F16),
    (INT8, 0, 4096, 1040, 9, BF16), (INT8, 0, 4097, 1040, 9, BF16),
    (INT8, 0, 500, 4112, 15, F32),      # eight column tiles
    (INT8, 0, 4096, 4096, 16, F16), (INT8, 0, 300, 4112, 16, F16),
    (INT8, 0, 64, 16384, 8, BF16), (INT8, 0, 64, 16400, 8, BF16),
    (UINT4, 128, 4736, 256, 17, F16), (UINT4, 128, 4737, 256, 17, F16), (UINT4, 128, 6144, 256, 32, BF16),
    (UINT4, 128, 8193, 256, 32, BF16), (INT4, 64, 4737, 320, 16, F16),
    (UINT4, 128, 4736, 1024, 32, F32), (UINT4, 128, 4737, 1024, 25, F32), (INT4, 128, 1000, 1024, 17, F32),
])
def test_canonical(qx, oracle_mod, layout, group, n, k, m, x_type):
    rng = np.random.Generator(np.random.Philox(key=[n * 31 + k, m * 7 + group]))
    weights, tensor = _tensor(qx, oracle_mod, rng, layout, group, n, k)
    x, x_exact = _storage((rng.standard_normal((m, k)) * 0.1).astype(np.float32), x_type)
    status, y = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK, qx.last_error()
    assert close(y, _product_f64(tensor, x_exact))
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()
