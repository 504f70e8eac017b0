"""Scratch of qx_lowbit_gemm_w8a8_dev counts every layout that a call of its size may put there, and nothing that none does."""

import pytest


def _up(value):
    return (value + 255) // 256 * 256


def _layouts(m, k):
    tiles = next(t for t in (1, 2, 4, 8) if m <= 8 * t)  # (eight rows of activations each)
    scales = _up(4 * m)
    rows = _up(m * k) + 2 * scales                       # dp4a kernel: codes, scales, sums
    streamed = _up((k + 63) // 64 * 512 * tiles) + 2 * scales
    return rows, streamed


# one to eight tiles of rows, rows of less than a step of 64 columns up to the longest
@pytest.mark.parametrize("k", [1, 63, 64, 65, 4096, 16512, 16513, 131000])
@pytest.mark.parametrize("m", [1, 2, 8, 9, 16, 17, 32, 33, 64])
def test_streamed_batches(qx, m, k):
    smaller = [_layouts(rows, k) for rows in range(1, m + 1)]
    assert qx.lib.qx_lowbit_w8a8_scratch_bytes(m, k) == max(max(layouts) for layouts in smaller)


def test_larger_batches_hold_the_streamed_ones(qx):
    for k in (1, 64, 4098, 131000):
        assert qx.lib.qx_lowbit_w8a8_scratch_bytes(65, k) >= qx.lib.qx_lowbit_w8a8_scratch_bytes(64, k)
