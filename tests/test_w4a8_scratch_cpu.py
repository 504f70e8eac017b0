"""Scratch of qx_lowbit_gemm_w8a8_dev: a size asked for once, for the largest batch and the longest row,
serves every smaller call (tests/test_w4a8_tensor_gpu.py runs such calls on one)."""

import pytest

ROWS = [1, 2, 4, 5, 12, 13, 32, 33, 64, 65, 100, 128, 129, 130, 256, 1000, 65535, 65536, 70000]
COLUMNS = [1, 31, 32, 33, 64, 1502, 4096, 4097, 4098, 4128, 16510, 16512, 16513, 16514, 16544, 131000]


def test_size_never_falls(qx):
    size = {(m, k): int(qx.lib.qx_lowbit_w8a8_scratch_bytes(m, k)) for m in ROWS for k in COLUMNS}
    for m, m_next in zip(ROWS, ROWS[1:]):
        assert all(size[m, k] <= size[m_next, k] for k in COLUMNS), (m, m_next)
    for k, k_next in zip(COLUMNS, COLUMNS[1:]):
        assert all(size[m, k] <= size[m, k_next] for m in ROWS), (k, k_next)


@pytest.mark.parametrize("m,k", [(0, 32), (4, 0), (-1, 32), (4, -32)])
def test_nothing_for_no_shape(qx, m, k):
    assert qx.lib.qx_lowbit_w8a8_scratch_bytes(m, k) == 0
