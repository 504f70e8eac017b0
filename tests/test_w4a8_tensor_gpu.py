"""W4A8 on the tensor cores (csrc/qx_scaled_gemm.cu from qx_lowbit_gemm_w8a8): f16 whole numbers with
sums below 2^24, so the result keeps every bit of the reference's
(tests/correctness/test_lowbit_w8a8.cpp:53-72 demands exact equality)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (2, 128, 258),      # smallest batch and matrix of rows that start on any byte
    (13, 128, 256),     # ... and of rows on whole vectors
    (4, 128, 258),      # the smallest of both above the lines of the small matrices
    (17, 128, 256),
    (1, 4096, 2050),    # one row of a large matrix
    (33, 129, 1033),    # an odd number of columns; a second tile of one row
    (64, 300, 2050),
    (65, 257, 1502),    # first large tile
    (130, 200, 1312),   # whole tiles only
    (5, 128, 16510),    # the longest rows of the tensor cores, and one step further: the integer kernel
    (5, 128, 16514),    # (sums up to the limit: test_sums_at_the_limit)
])
def test_bits_of_the_reference(qx, orc, m, n, k):
    rng = np.random.Generator(np.random.Philox(key=[m * 1000 + n, k]))
    packed = rng.integers(0, 256, (n, (k + 1) // 2), dtype=np.uint8)
    scales = rng.uniform(0.001, 0.1, n).astype(np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    x[m // 2, ::5] = 0.0
    status, y = qx.lowbit_gemm_w8a8(packed.reshape(-1), scales, x, m, n, k)
    assert status == qx.OK, qx.last_error()
    _, want = orc.lowbit_gemm_w8a8(packed.reshape(-1), scales, x, m, n, k)
    assert np.array_equal(np.asarray(y).view(np.uint32).reshape(m, n), np.asarray(want).view(np.uint32).reshape(m, n))
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()


@pytest.mark.parametrize("k", [16510, 16512, 20001])
def test_sums_at_the_limit(qx, orc, k):
    """Products of -8 * 127 behind a few of 1 * 127: odd sums just below 2^24, which lose their last bit as
    soon as f32 or the tensor core rounds anything, and sums beyond it for the integer kernel."""
    m, n = 20, 130
    column, row = np.arange(k + k % 2)[None, :], np.arange(n)[:, None]
    nibbles = np.where(column < 2 * (row % 8) + 1, 9, 0).astype(np.uint8)  # odd numbers of early columns
    if k > 16512:
        nibbles[(column >= 256) & (column % 128 == 7) & (column % (256 + 128 * (row % 5)) < 128)] = 9
    packed = np.ascontiguousarray(nibbles[:, 0::2] | (nibbles[:, 1::2] << 4))
    scales = np.full(n, 0.5, np.float32)
    x = np.ones((m, k), np.float32)
    dots = 127 * (nibbles[:, :k].astype(np.int64) - 8).sum(axis=1)
    parts = np.add.reduceat((nibbles[:, :k].astype(np.int64) - 8) * 127, np.arange(0, k, 128), axis=1)
    chain = np.add.accumulate(parts.astype(np.float32), axis=1, dtype=np.float32)[:, -1]
    if k <= 16512:
        assert np.all((np.abs(dots) > 1 << 23) & (np.abs(dots) < 1 << 24) & (dots % 2 == 1))
    else:  # f32 sums of 128 columns would end elsewhere
        assert np.any(chain != dots.astype(np.float32))
    status, y = qx.lowbit_gemm_w8a8(packed.reshape(-1), scales, x, m, n, k)
    assert status == qx.OK, qx.last_error()
    _, want = orc.lowbit_gemm_w8a8(packed.reshape(-1), scales, x, m, n, k)
    assert np.array_equal(want[0], dots.astype(np.float32) * np.float32(0.5) * (np.float32(1.0) / np.float32(127.0)))
    assert np.array_equal(np.asarray(y).view(np.uint32).reshape(m, n), np.asarray(want).view(np.uint32).reshape(m, n))


def _exact(orc, packed, scales, x, m, n, k):
    """float(dot) * weight scale * activation scale on the oracle's codes; the dots in float64,
    where they are exact, as the oracle's own loop takes seconds on these sizes."""
    _, codes, xs = orc.quantize_int8(x, m, k, 0)
    rows = packed.reshape(n, -1)
    w = np.stack((rows & 15, rows >> 4), axis=-1).reshape(n, -1)[:, :k].astype(np.float64) - 8.0
    dot = (codes.reshape(m, k).astype(np.float64) @ w.T).astype(np.float32)
    return (dot * scales[None, :]) * xs.reshape(m, 1)


def _twice_on_one_scratch(qx, packed, scales, x, m, n, k, fill=255):
    """Two calls of the device entry point on the same scratch, full of `fill` before the first."""
    import torch
    scratch = torch.full((int(qx.lib.qx_lowbit_w8a8_scratch_bytes(m, k)),), fill, dtype=torch.uint8, device="cuda")
    w, ws, xd = (torch.from_numpy(a).cuda() for a in (packed, scales, x))
    results = []
    for _ in range(2):
        y = torch.full((m, n), np.nan, device="cuda")
        torch.cuda.synchronize()
        status = qx.lib.qx_lowbit_gemm_w8a8_dev(w.data_ptr(), ws.data_ptr(), xd.data_ptr(), y.data_ptr(),
                                                scratch.data_ptr(), m, n, k, torch.cuda.current_stream().cuda_stream)
        assert status == qx.OK, qx.last_error()
        torch.cuda.synchronize()
        results.append(y.cpu().numpy())
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()
    return results


# Odd numbers of 128-column stages at the end of a tile, and CTAs that go on to the next tile behind
# it: two groups of converter warps share rings of two stages (33 .. 64 rows that start on any byte)
@pytest.mark.parametrize("m,n,k", [(33, 4096, 4098), (64, 14336, 1154), (48, 25600, 100), (40, 20000, 354)])
def test_odd_stages_across_tiles(qx, orc, m, n, k):
    rng = np.random.Generator(np.random.Philox(key=[m, n + k]))
    packed = rng.integers(0, 256, (n, (k + 1) // 2), dtype=np.uint8)
    scales = rng.uniform(0.001, 0.1, n).astype(np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    want = _exact(orc, packed, scales, x, m, n, k)
    for y in _twice_on_one_scratch(qx, packed, scales, x, m, n, k):
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))


# tiles cut into pieces on a full grid, so that every CTA's counters are used: 16 epilogue warps
# from 65 rows on, 8 below
@pytest.mark.parametrize("m,n,k", [(64, 4096, 4096), (65, 4096, 4096), (100, 4096, 4098), (128, 14336, 4096)])
def test_pieces_of_a_full_grid(qx, orc, m, n, k):
    rng = np.random.Generator(np.random.Philox(key=[m, n + k]))
    packed = rng.integers(0, 256, (n, (k + 1) // 2), dtype=np.uint8)
    scales = rng.uniform(0.001, 0.1, n).astype(np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    want = _exact(orc, packed, scales, x, m, n, k)
    for y in _twice_on_one_scratch(qx, packed, scales, x, m, n, k):
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))


def test_scratch_of_the_largest_call_serves_smaller_ones(qx, orc):
    import torch
    n, guard = 4096, 32 << 20
    size = int(qx.lib.qx_lowbit_w8a8_scratch_bytes(256, 4098))
    scratch = torch.full((size + guard,), 0xA5, dtype=torch.uint8, device="cuda")
    rng = np.random.Generator(np.random.Philox(key=[11, 12]))
    for m, k in [(256, 4098), (128, 4096), (64, 4098), (5, 4096), (1, 2050)]:
        packed = rng.integers(0, 256, (n, (k + 1) // 2), dtype=np.uint8)
        scales = rng.uniform(0.001, 0.1, n).astype(np.float32)
        x = rng.standard_normal((m, k)).astype(np.float32)
        w, ws, xd = (torch.from_numpy(a).cuda() for a in (packed, scales, x))
        y = torch.full((m, n), np.nan, device="cuda")
        torch.cuda.synchronize()
        status = qx.lib.qx_lowbit_gemm_w8a8_dev(w.data_ptr(), ws.data_ptr(), xd.data_ptr(), y.data_ptr(),
                                                scratch.data_ptr(), m, n, k, torch.cuda.current_stream().cuda_stream)
        assert status == qx.OK, qx.last_error()
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy().view(np.uint32), _exact(orc, packed, scales, x, m, n, k).view(np.uint32))
        assert bool((scratch[size:] == 0xA5).all())


# Weights written by the kernel directly in front, other ones on every call: nothing of them may be
# fetched before that kernel is done (dp4a kernel, tensor cores with rows on vectors and on any byte)
@pytest.mark.parametrize("m,n,k", [(1, 14336, 4096), (8, 4096, 4096), (32, 8192, 4096), (16, 8192, 4098)])
def test_weights_written_in_front(qx, orc, m, n, k):
    import torch
    rng = np.random.Generator(np.random.Philox(key=[m, n, k][:2]))
    sides = [torch.from_numpy(rng.integers(0, 256, (n, k // 2), dtype=np.uint8)).cuda() for _ in range(2)]
    scales = rng.uniform(0.001, 0.1, n).astype(np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    want = [torch.from_numpy(_exact(orc, side.cpu().numpy(), scales, x, m, n, k)).cuda() for side in sides]
    scratch = torch.zeros(int(qx.lib.qx_lowbit_w8a8_scratch_bytes(m, k)), dtype=torch.uint8, device="cuda")
    w, ws, xd = torch.zeros_like(sides[0]), torch.from_numpy(scales).cuda(), torch.from_numpy(x).cuda()
    outputs = [torch.full((m, n), np.nan, device="cuda") for _ in range(20)]
    torch.cuda.synchronize()
    for i, y in enumerate(outputs):
        torch.bitwise_xor(sides[i % 2], 0, out=w)
        status = qx.lib.qx_lowbit_gemm_w8a8_dev(w.data_ptr(), ws.data_ptr(), xd.data_ptr(), y.data_ptr(),
                                                scratch.data_ptr(), m, n, k, torch.cuda.current_stream().cuda_stream)
        assert status == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    for i, y in enumerate(outputs):
        assert torch.equal(y, want[i % 2]), i
