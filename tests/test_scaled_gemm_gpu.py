"""Batched projections on the tensor cores with scales along K (csrc/qx_scaled_gemm.cu), through
the C ABI: canonical int4 / uint4 / int8 tensors and q8_0 panels with 16-bit activations.

Every product is exact and every group is scaled in f32, so the tolerance is that of f32 sums, the
rule of the reference's own projection test: 4e-5 * (1 + |exact|) against float64.
"""

import numpy as np
import pytest

from test_canonical_gpu import BF16, F16, F32, INT4, INT8, OUT_TOLERANCE, UINT4, activation_f64, close, widen

pytestmark = pytest.mark.gpu

GROUP, CHANNEL = 4, 3


def _storage(x, x_type):
    """(activations as the entry point takes them, the same values as f32)"""
    import torch
    if x_type == F32:
        return x, x
    t = torch.from_numpy(x).to(torch.float16 if x_type == F16 else torch.bfloat16)
    return np.ascontiguousarray(t.view(torch.int16).numpy().view(np.uint16)), t.float().numpy()


def _tensor(qx, oracle_mod, rng, layout, group, n, k, act_order=None):
    groups = k // group if group else 1
    mode = GROUP if group else CHANNEL
    codes = n * k if layout == INT8 else n * k // 2
    data = rng.integers(0, 256, codes, dtype=np.uint8)
    scales = rng.uniform(0.002, 0.03, n * groups).astype(np.float32)
    zeros = rng.integers(0, 16, n * groups).astype(np.float32) if layout == UINT4 else None
    view = qx.canonical_view(layout, mode, n, k, group or k, data, scales, zeros=zeros, act_order=act_order)
    weights = qx.CanonicalWeights()
    assert weights.prepare(view) == qx.OK, qx.last_error()
    return weights, oracle_mod.CanonicalTensor(layout, mode, n, k, group or k, data, scales, zeros, None, act_order)


def _product_f64(tensor, x):
    """The product in float64 by one matrix product: the oracle's loop takes seconds on large matrices."""
    data = np.asarray(tensor.data).reshape(-1).view(np.uint8)
    if tensor.layout == INT8:
        q = data.view(np.int8).astype(np.float64)
    else:
        q = np.stack((data & 15, data >> 4), axis=-1).reshape(-1).astype(np.float64)
        if tensor.layout == INT4:
            q = np.where(q >= 8, q - 16, q)
    q = q.reshape(tensor.rows, -1, tensor.group_size)
    groups = (tensor.rows, q.shape[1], 1)
    if tensor.zeros is not None:
        q = q - np.asarray(tensor.zeros, np.float64).reshape(groups)
    w = (q * np.asarray(tensor.scales, np.float64).reshape(groups)).reshape(tensor.rows, -1)
    return x.astype(np.float64) @ w.T


@pytest.mark.parametrize("layout,group,n,k,m,x_type", [
    (UINT4, 128, 4097, 2048, 5, BF16),   # smallest batch, a last tile of one row
    (UINT4, 128, 1025, 1152, 32, F16),   # half a slab at the end
    (INT4, 32, 1000, 1056, 33, BF16),    # 33 groups: the last stage holds groups of padding
    (UINT4, 32, 1100, 992, 64, F32),     # three planes, largest small tile
    (INT4, 64, 260, 2112, 65, F16),      # first large tile
    (UINT4, 96, 256, 1152, 130, BF16),   # groups that do not divide a slab
    (INT4, 0, 384, 800, 257, F32),       # one scale per row, tokens in five tiles
    (UINT4, 256, 640, 2560, 300, BF16),  # groups larger than an accumulator's columns
    (INT8, 64, 900, 1088, 70, F32),      # bytes: half a slot at the end
    (INT8, 0, 4100, 2064, 512, BF16),    # bytes with one scale per row: rows of 129 vectors
])
def test_batches_against_float64(qx, orc, oracle_mod, layout, group, n, k, m, x_type):
    rng = np.random.Generator(np.random.Philox(key=[n * 31 + k, m * 7 + group]))
    weights, tensor = _tensor(qx, oracle_mod, rng, layout, group, n, k)
    x, x_exact = _storage((rng.standard_normal((m, k)) * 0.1).astype(np.float32), x_type)
    bias = rng.standard_normal(n).astype(np.float32)
    exact = orc.canonical_gemm_f64(tensor, np.ascontiguousarray(x_exact), F32, m)
    status, y = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK, qx.last_error()
    assert close(y, exact)
    status, typed = weights.qgemm_storage(x, x_type, m, y_type=BF16, bias=bias, activation=3)
    assert status == qx.OK, qx.last_error()
    assert close(widen(typed, BF16), activation_f64(exact + bias.astype(np.float64)[None, :], 3), OUT_TOLERANCE[BF16])
    status, again = weights.qgemm_storage(x, x_type, m)  # pieces of a tile are added in a fixed order
    assert status == qx.OK and np.array_equal(again.view(np.uint32), y.view(np.uint32))
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()


# The same edges above the lines at which the tensor cores take over
@pytest.mark.parametrize("layout,group,n,k,m,x_type", [
    (UINT4, 128, 4097, 4096, 5, BF16),   # smallest batch, a last tile of one row
    (INT4, 32, 4001, 1056, 33, BF16),    # 33 groups: the last stage holds groups of padding
    (UINT4, 32, 2300, 992, 64, F32),     # three planes, largest small tile
    (INT4, 64, 1030, 2112, 65, F16),     # first large tile
    (UINT4, 96, 1010, 1152, 130, BF16),  # groups that do not divide a slab
    (INT4, 0, 700, 800, 257, F32),       # one scale per row, tokens in five tiles
    (UINT4, 128, 130, 8192, 128, F16),   # two tiles in pieces of one slab each
    (INT8, 64, 2000, 1088, 70, F32),     # bytes: half a slot at the end
    (UINT4, 128, 14336, 1024, 512, BF16),  # several rounds of tiles on every SM
])
def test_edges_above_the_lines(qx, orc, oracle_mod, layout, group, n, k, m, x_type):
    rng = np.random.Generator(np.random.Philox(key=[n * 31 + k, m * 7 + group]))
    weights, tensor = _tensor(qx, oracle_mod, rng, layout, group, n, k)
    x, x_exact = _storage((rng.standard_normal((m, k)) * 0.1).astype(np.float32), x_type)
    exact = _product_f64(tensor, x_exact)
    status, y = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK, qx.last_error()
    assert close(y, exact)
    status, again = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK and np.array_equal(again.view(np.uint32), y.view(np.uint32))
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()


# Tiles that end on an odd number of 128-column stages, CTAs that go on to the next tile, rings of two
# stages or two slots: f32 activations (three planes) of more than 32 tokens, bytes of 25 to 32
@pytest.mark.parametrize("layout,group,n,k,m,x_type", [
    (UINT4, 128, 4096, 4224, 64, F32),
    (INT4, 64, 14336, 1152, 40, F32),
    (INT8, 64, 12800, 1152, 28, F32),
    (INT8, 128, 9000, 896, 60, F32),
    (UINT4, 32, 25600, 96, 32, BF16),    # tiles of a single stage
])
def test_odd_stages_across_tiles(qx, orc, oracle_mod, layout, group, n, k, m, x_type):
    rng = np.random.Generator(np.random.Philox(key=[n + k, m + group]))
    weights, tensor = _tensor(qx, oracle_mod, rng, layout, group, n, k)
    x, x_exact = _storage((rng.standard_normal((m, k)) * 0.1).astype(np.float32), x_type)
    exact = _product_f64(tensor, x_exact)
    status, first = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK, qx.last_error()
    assert close(first, exact)
    for _ in range(5):
        status, y = weights.qgemm_storage(x, x_type, m)
        assert status == qx.OK and np.array_equal(y.view(np.uint32), first.view(np.uint32))
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()


@pytest.mark.parametrize("n", [900, 1100])  # the digit kernels, the tensor cores
def test_act_order_and_unaligned_activations(qx, orc, oracle_mod, n):
    import torch
    k, m = 1024, 40
    rng = np.random.Generator(np.random.Philox(key=[5, 6]))
    order = rng.permutation(k).astype(np.int32)
    weights, tensor = _tensor(qx, oracle_mod, rng, INT4, 128, n, k, act_order=order)
    plain, plain_tensor = _tensor(qx, oracle_mod, rng, INT4, 128, n, k)
    x, x_exact = _storage((rng.standard_normal((m, k)) * 0.1).astype(np.float32), BF16)
    status, y = weights.qgemm_storage(x, BF16, m)
    assert status == qx.OK, qx.last_error()
    assert close(y, orc.canonical_gemm_f64(tensor, np.ascontiguousarray(x_exact), F32, m))
    # device activations that start two bytes past a 16-byte boundary
    buffer = torch.zeros(m * k + 8, dtype=torch.int16, device="cuda")
    shifted = buffer[1:1 + m * k].view(m, k)
    shifted.copy_(torch.from_numpy(x.view(np.int16)))
    out = torch.zeros((m, n), device="cuda")
    assert plain.qgemm_storage_dev(shifted, BF16, out, F32, m) == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    assert close(out.cpu().numpy(), orc.canonical_gemm_f64(plain_tensor, np.ascontiguousarray(x_exact), F32, m))


@pytest.mark.parametrize("n,k,m", [(2048, 1024, 33), (4096, 1024, 40)])  # (f32: digit kernels, tensor cores)
def test_a_token_that_is_not_finite_stays_alone(qx, orc, oracle_mod, n, k, m):
    rng = np.random.Generator(np.random.Philox(key=[8, 9]))
    weights, tensor = _tensor(qx, oracle_mod, rng, UINT4, 64, n, k)
    x = (rng.standard_normal((m, k)) * 0.1).astype(np.float32)
    x[4, 17] = np.nan
    for x_type in (F32, BF16):
        stored, values = _storage(x, x_type)
        status, y = weights.qgemm_storage(stored, x_type, m)
        assert status == qx.OK, qx.last_error()
        assert np.all(np.isnan(y[4]))
        finite = [r for r in range(m) if r != 4]
        exact = orc.canonical_gemm_f64(tensor, np.ascontiguousarray(values[finite]), F32, m - 1)
        assert close(y[finite], exact)


# Activations near the ends of their type's range: a group's sum of whole weights times activations
# is far beyond f32 where the scaled result is not, and down to the smallest normal numbers
@pytest.mark.parametrize("layout,group,n,k,m,x_type,size", [
    (UINT4, 128, 1100, 1024, 64, BF16, 1e37), (UINT4, 128, 1100, 1024, 64, BF16, 1e-36),
    (INT8, 128, 2048, 1024, 100, BF16, 1e36), (INT8, 128, 2048, 1024, 100, BF16, 1e-36),
    (INT4, 32, 4096, 1024, 40, F32, 2e37), (INT4, 32, 4096, 1024, 40, F32, 1e-28)])
def test_activations_of_extreme_size(qx, oracle_mod, layout, group, n, k, m, x_type, size):
    rng = np.random.Generator(np.random.Philox(key=[n + k, m + group]))
    weights, tensor = _tensor(qx, oracle_mod, rng, layout, group, n, k)
    x, x_exact = _storage((rng.standard_normal((m, k)) * size).astype(np.float32), x_type)
    exact = _product_f64(tensor, x_exact)
    status, y = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK, qx.last_error()
    assert np.all(np.isfinite(y))
    # (1e-5: far above f32 sums, far below one overflow or a lost plane)
    assert np.linalg.norm((y - exact) / size) <= 1e-5 * np.linalg.norm(exact / size)


@pytest.mark.parametrize("size", [1e36, 1e-30])
def test_q8_0_prefill_of_extreme_size(qx, orc, wl, size):
    import torch
    n, k, m = 512, 1024, 40
    packed = wl.packed_blocks(0, n, k, 0.001, 0.02, seed=9)
    xb = wl.to_bf16_bits(wl.activations_f32(m, k, seed=m) * np.float32(size))
    weights = qx.PackedWeights()
    assert weights.prepare(0, packed, n, k) == qx.OK, qx.last_error()
    y = torch.zeros((m, n), device="cuda")
    assert weights.qgemm_bf16_dev(torch.from_numpy(xb.view(np.int16)).cuda(), y, m) == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    _, exact = orc.qgemm_f64(0, packed, wl.bf16_bits_to_f32(xb), m, n, k)
    got = y.cpu().numpy().astype(np.float64)
    assert np.all(np.isfinite(got))
    assert np.linalg.norm((got - exact) / size) <= 1e-5 * np.linalg.norm(exact / size)


@pytest.mark.parametrize("x_type", [F32, F16, BF16])
def test_an_infinite_activation(qx, oracle_mod, x_type):
    """16-bit types: an infinity of the weight's sign, or NaN where the weight is zero, as the reference's
    sums give; f32: NaN in the whole token. Other tokens do not see it."""
    n, k, m = 4096, 1024, 40
    rng = np.random.Generator(np.random.Philox(key=[18, 19]))
    weights, tensor = _tensor(qx, oracle_mod, rng, UINT4, 64, n, k)
    x = (rng.standard_normal((m, k)) * 0.1).astype(np.float32)
    x[7, 100] = np.inf
    stored, values = _storage(x, x_type)
    status, y = weights.qgemm_storage(stored, x_type, m)
    assert status == qx.OK, qx.last_error()
    finite = [r for r in range(m) if r != 7]
    assert close(y[finite], _product_f64(tensor, values[finite]))
    if x_type == F32:
        assert np.all(np.isnan(y[7]))
    else:
        column = np.zeros((1, k), np.float32)
        column[0, 100] = 1.0
        weight = _product_f64(tensor, column)[0]
        assert np.array_equal(y[7] == np.inf, weight > 0) and np.array_equal(y[7] == -np.inf, weight < 0)
        assert np.array_equal(np.isnan(y[7]), weight == 0)


@pytest.mark.parametrize("n,k,m", [(128, 256, 16), (300, 1056, 33), (257, 416, 64), (640, 2080, 65), (384, 11008, 331)])
def test_q8_0_prefill(qx, orc, wl, n, k, m):
    import torch
    packed = wl.packed_blocks(0, n, k, 0.001, 0.02, seed=n + k)
    xb = wl.to_bf16_bits(wl.activations_f32(m, k, seed=m))
    weights = qx.PackedWeights()
    assert weights.prepare(0, packed, n, k) == qx.OK, qx.last_error()
    y = torch.full((m, n + 3), -7.0, device="cuda")  # a row stride of its own
    status = weights.qgemm_bf16_dev(torch.from_numpy(xb.view(np.int16)).cuda(), y, m, ldy=n + 3)
    assert status == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    got = y.cpu().numpy()
    assert np.all(got[:, n:] == -7.0)
    _, exact = orc.qgemm_f64(0, packed, wl.bf16_bits_to_f32(xb), m, n, k)
    # K terms of f32 sums: at most K / 32 roundings of 2^-24 of the running sum, which stays below
    # the sum of the magnitudes; 4e-6 of a row's rms is four times what is measured
    rms = np.sqrt((exact ** 2).mean(axis=1, keepdims=True))
    assert np.all(np.abs(got[:, :n] - exact) <= 4e-6 * (np.abs(exact) + rms))
