"""W8A8 on the tensor cores over the tiles that its rule chooses: 32 to 256 tokens, 128 or 256 channels, up to eight
K-slabs in flight. Exact sums, so the result has the reference's bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (33, 128, 1040),     # one and a bit tiles of 32 tokens, nine slabs in a ring of eight
    (64, 8193, 128),     # one slab, a last tile of one channel
    (97, 4000, 272),
    (128, 4096, 2064),   # 128 tiles of 32 tokens
    (200, 2048, 1024),
    (257, 300, 528),
    (300, 14336, 144),   # 256 channels x 160 tokens
    (1300, 9000, 256),   # several rounds of tiles
])
def test_tiles(qx, m, n, k):
    rng = np.random.Generator(np.random.Philox(key=[m, n + k]))
    w, x = rng.integers(-128, 128, (n, k), dtype=np.int8), rng.integers(-128, 128, (m, k), dtype=np.int8)
    ws, xs = rng.uniform(0.001, 0.01, n).astype(np.float32), rng.uniform(0.005, 0.05, m).astype(np.float32)
    status, y = qx.int8_gemm(w, x, ws, xs, m, n, k)
    assert status == qx.OK, qx.last_error()
    want = ((x.astype(np.float64) @ w.astype(np.float64).T).astype(np.float32) * ws[None, :]) * xs[:, None]
    assert np.array_equal(y.view(np.uint32), want.view(np.uint32))
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()
