"""The tcgen05 kernels of csrc/qx_scaled_gemm.cu beyond the batches that stream their codes (csrc/qx_stream_mma.cu):
exact f32 sums of W4A8, odd numbers of stages in tiles behind one another, the small tiles of canonical batches."""

import numpy as np
import pytest

from test_canonical_gpu import BF16, F16, F32, INT4, INT8, UINT4, close
from test_scaled_gemm_gpu import _product_f64, _storage, _tensor
from test_w4a8_tensor_gpu import _exact, _twice_on_one_scratch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [65, 130])
@pytest.mark.parametrize("k", [16510, 16512, 20001])
def test_w4a8_sums_at_the_limit(qx, orc, m, k):
    """Products of -8 * 127 behind a few of 1 * 127: odd sums just below 2^24, which lose their last bit as
    soon as f32 or the tensor core rounds anything; and longer rows, which the integer kernel takes."""
    n = 130
    column, row = np.arange(k + k % 2)[None, :], np.arange(n)[:, None]
    nibbles = np.where(column < 2 * (row % 8) + 1, 9, 0).astype(np.uint8)
    packed = np.ascontiguousarray(nibbles[:, 0::2] | (nibbles[:, 1::2] << 4))
    scales = np.full(n, 0.5, np.float32)
    dots = 127 * (nibbles[:, :k].astype(np.int64) - 8).sum(axis=1)
    if k <= 16512:
        assert np.all((np.abs(dots) > 1 << 23) & (np.abs(dots) < 1 << 24) & (dots % 2 == 1))
    want = np.tile(dots.astype(np.float32) * np.float32(0.5) * (np.float32(1.0) / np.float32(127.0)), (m, 1))
    for y in _twice_on_one_scratch(qx, packed, scales, np.ones((m, k), np.float32), m, n, k):
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))


# odd numbers of 128-column stages at the end of a tile, and CTAs that go on to the next tile behind it; rows on whole
# vectors and on any byte, whole tiles and pieces
@pytest.mark.parametrize("m,n,k", [(65, 4096, 4098), (128, 14336, 1154), (129, 25600, 100), (90, 20000, 354), (70, 14336, 1120)])
def test_w4a8_odd_stages_across_tiles(qx, orc, m, n, k):
    rng = np.random.Generator(np.random.Philox(key=[m, n + k]))
    packed = rng.integers(0, 256, (n, (k + 1) // 2), dtype=np.uint8)
    scales = rng.uniform(0.001, 0.1, n).astype(np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    want = _exact(orc, packed, scales, x, m, n, k)
    for y in _twice_on_one_scratch(qx, packed, scales, x, m, n, k):
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))


# Tiles of 32 and 64 tokens: two groups of converter warps take the stages in turn. Odd numbers of stages, more tiles than
# SMs, pieces of tiles; the smallest batches that do not stream.
@pytest.mark.parametrize("layout,group,n,k,m,x_type", [
    (UINT4, 128, 14336, 1152, 33, F16),   # nine stages, 112 tiles
    (INT4, 128, 25600, 128, 48, BF16),    # one stage, 200 tiles
    (INT4, 32, 9000, 1056, 20, BF16),     # groups of 32 above 16 tokens
    (UINT4, 128, 16400, 640, 17, F16),    # 17 tokens on more rows than stream with them
    (INT8, 64, 20000, 320, 40, BF16),     # bytes: five half stages
    (UINT4, 64, 4096, 4160, 64, F32),     # three planes
])
def test_small_tiles_across_tiles(qx, oracle_mod, layout, group, n, k, m, x_type):
    rng = np.random.Generator(np.random.Philox(key=[n * 31 + k, m * 7 + group]))
    weights, tensor = _tensor(qx, oracle_mod, rng, layout, group, n, k)
    x, x_exact = _storage((rng.standard_normal((m, k)) * 0.1).astype(np.float32), x_type)
    status, y = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK, qx.last_error()
    assert close(y, _product_f64(tensor, x_exact))
    status, again = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK and np.array_equal(again.view(np.uint32), y.view(np.uint32))
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()
