"""Small batches whose codes are streamed past the activations (csrc/qx_stream_mma.cu), through the C ABI: W8A8
and W4A8 bit for bit, canonical tensors against float64 within the reference test's own 4e-5 * (1 + |exact|)."""

import numpy as np
import pytest

from test_canonical_gpu import BF16, F16, F32, INT4, INT8, OUT_TOLERANCE, UINT4, activation_f64, close, widen
from test_scaled_gemm_gpu import CHANNEL, _product_f64, _storage, _tensor
from test_w4a8_tensor_gpu import _exact

pytestmark = pytest.mark.gpu


# tails of a step (64 columns) of 16, 32 and 48; fewer steps than warps; last tiles of 1 .. 16 rows; one to
# eight column tiles; one and two tiles of rows per warp (from 6144 rows on)
@pytest.mark.parametrize("azp", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 1, 16), (4, 17, 1424), (8, 33, 96), (9, 6145, 112), (16, 6160, 512), (17, 1000, 2064),
                                   (32, 6200, 80), (31, 31, 4096)])
def test_w8a8(qx, m, n, k, azp):
    rng = np.random.Generator(np.random.Philox(key=[m * 7 + n, k]))
    w = rng.integers(-128, 128, (n, k), dtype=np.int8)
    x = rng.integers(-128, 128, (m, k), dtype=np.int8)
    ws, xs = rng.uniform(0.001, 0.01, n).astype(np.float32), rng.uniform(0.005, 0.05, m).astype(np.float32)
    row_sum, zp = w.sum(axis=1, dtype=np.int32), rng.integers(-20, 21, m, dtype=np.int32)
    acc = x.astype(np.float64) @ w.astype(np.float64).T
    if azp:
        acc -= zp.astype(np.float64)[:, None] * row_sum.astype(np.float64)[None, :]
        status, y = qx.int8_gemm(w, x, ws, xs, m, n, k, row_sum=row_sum, zp=zp, asymmetric=True)
    else:
        status, y = qx.int8_gemm(w, x, ws, xs, m, n, k)
    assert status == qx.OK, qx.last_error()
    want = (acc.astype(np.float32) * ws[None, :]) * xs[:, None]
    assert np.array_equal(y.view(np.uint32), want.view(np.uint32))


# rows on whole vectors and on any byte (k of every remainder, packed rows from an odd address on): nothing in front of
# or behind the packed rows is used, whatever it holds
@pytest.mark.parametrize("offset", [0, 1, 8, 13])
@pytest.mark.parametrize("m,n,k", [(1, 1, 2), (1, 300, 33), (3, 17, 1024), (8, 130, 1031), (16, 6161, 130), (31, 64, 4098),
                                   (33, 6145, 96), (64, 515, 2047)])
def test_w4a8(qx, orc, m, n, k, offset):
    import torch
    rng = np.random.Generator(np.random.Philox(key=[m * 5 + n, k * 16 + offset]))
    packed = rng.integers(0, 256, (n, (k + 1) // 2), dtype=np.uint8)
    scales = rng.uniform(0.001, 0.1, n).astype(np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    want = _exact(orc, packed, scales, x, m, n, k)
    block = torch.full((packed.size + offset,), 255, dtype=torch.uint8, device="cuda")
    block[offset:offset + packed.size] = torch.from_numpy(packed.reshape(-1)).cuda()
    ws, xd = torch.from_numpy(scales).cuda(), torch.from_numpy(x).cuda()
    scratch = torch.full((int(qx.lib.qx_lowbit_w8a8_scratch_bytes(m, k)),), 255, dtype=torch.uint8, device="cuda")
    y = torch.full((m, n), np.nan, device="cuda")
    assert qx.lib.qx_lowbit_gemm_w8a8_dev(block.data_ptr() + offset, ws.data_ptr(), xd.data_ptr(), y.data_ptr(),
                                          scratch.data_ptr(), m, n, k, torch.cuda.current_stream().cuda_stream) == qx.OK
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("layout,group,n,k,m,x_type", [
    (INT8, 0, 262145, 16, 1, BF16),      # digits: one step, one warp with work, a last tile of one row
    (INT8, 0, 6161, 1072, 2, F16),       # two tiles of rows per warp, a tail of 48 columns
    (INT8, 0, 500, 4112, 16, F32),       # eight column tiles
    (UINT4, 128, 6569, 128, 5, F16),     # one group
    (UINT4, 128, 6145, 1152, 8, BF16),   # rows as they are, two tiles of rows
    (UINT4, 128, 6145, 1152, 9, F16),    # in fragments
    (INT4, 96, 260, 1056, 16, BF16),     # groups of three steps, act-order
    (INT4, 32, 4097, 2080, 16, F16),     # chains of four and a rest
    (UINT4, 64, 4096, 4160, 5, F32),     # three planes
    (INT4, 0, 4096, 1312, 24, F32),      # one scale per row, a last step of 32 columns
    (INT8, 64, 1000, 1088, 17, F16),     # bytes: sums of 32 columns
    (INT8, 160, 6200, 1120, 7, BF16),
    (INT8, 128, 2048, 2048, 31, F32),
])
def test_canonical(qx, oracle_mod, layout, group, n, k, m, x_type):
    rng = np.random.Generator(np.random.Philox(key=[n * 31 + k, m * 7 + group]))
    order = rng.permutation(k).astype(np.int32) if layout == INT4 and group == 96 else None
    weights, tensor = _tensor(qx, oracle_mod, rng, layout, group, n, k, act_order=order)
    x, x_exact = _storage((rng.standard_normal((m, k)) * 0.1).astype(np.float32), x_type)
    exact = _product_f64(tensor, x_exact if order is None else x_exact[:, order])
    bias = rng.standard_normal(n).astype(np.float32)
    status, y = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK, qx.last_error()
    assert close(y, exact)
    status, typed = weights.qgemm_storage(x, x_type, m, y_type=BF16, bias=bias, activation=3)
    assert status == qx.OK, qx.last_error()
    assert close(widen(typed, BF16), activation_f64(exact + bias.astype(np.float64)[None, :], 3), OUT_TOLERANCE[BF16])


# An activation far above the others of its token, met by codes of zero in its 16 columns: the others keep the bits that
# they have without it. 2^-24 of the result: one rounding each, and fixed-point steps of 2^-31 below the others. (A token of
# size 1e35 gives results of up to 5e37; f32 ends at 3.4e38.)
@pytest.mark.parametrize("m,x_type,size,outlier", [
    (1, BF16, 1.0, 0.0), (1, BF16, 1.0, 2.0 ** 10), (4, BF16, 1.0, 2.0 ** 20), (1, F32, 1.0, 2.0 ** 26), (3, F32, 1.0, 2.0 ** 60),
    (2, F16, 0.01, 2.0 ** 15), (1, BF16, 1e-25, 0.0), (4, F32, 1e-33, 0.0), (2, F32, 1e-20, 1e10), (1, F32, 1e35, 0.0)])
def test_a_wide_range_within_a_token(qx, m, x_type, size, outlier):
    n, k, column = 2048, 4096, 1000
    rng = np.random.Generator(np.random.Philox(key=[n + m, int(outlier % 1000)]))
    codes = rng.integers(-127, 128, (n, k), dtype=np.int8)
    codes[:, column // 16 * 16:column // 16 * 16 + 16] = 0
    scales = rng.uniform(0.002, 0.03, n).astype(np.float32)
    weights = qx.CanonicalWeights()
    view = qx.canonical_view(INT8, CHANNEL, n, k, k, codes.view(np.uint8).reshape(-1), scales)
    assert weights.prepare(view) == qx.OK, qx.last_error()
    values = (rng.standard_normal((m, k)) * size).astype(np.float32)
    if outlier:
        values[:, column] = outlier
    x, x_exact = _storage(values, x_type)
    exact = (x_exact.astype(np.float64) @ codes.astype(np.float64).T) * scales.astype(np.float64)
    status, y = weights.qgemm_storage(x, x_type, m)
    assert status == qx.OK, qx.last_error()
    error = np.linalg.norm((y - exact) / size, axis=1) / np.linalg.norm(exact / size, axis=1)
    assert np.all(error <= 2.0 ** -24), error


# below, at and above the line of the streamed route; rows whose digits outgrow the small scratch
@pytest.mark.parametrize("n,k", [(256, 1024), (1023, 1024), (1024, 1024), (1500, 2048), (2048, 2048), (32, 40000)])
def test_one_to_four_tokens_have_the_bits_of_one(qx, oracle_mod, n, k):
    rng = np.random.Generator(np.random.Philox(key=[n, k]))
    weights, _ = _tensor(qx, oracle_mod, rng, INT8, 0, n, k)
    x, _ = _storage(rng.standard_normal((4, k)).astype(np.float32), BF16)
    single = [weights.qgemm_storage(x[i:i + 1], BF16, 1)[1][0] for i in range(4)]
    for m in (2, 3, 4):
        status, y = weights.qgemm_storage(x[:m], BF16, m)
        assert status == qx.OK, qx.last_error()
        assert all(np.array_equal(y[i].view(np.uint32), single[i].view(np.uint32)) for i in range(m)), m


@pytest.mark.parametrize("layout,group", [(INT8, 0), (UINT4, 128)])
def test_values_that_are_not_finite(qx, oracle_mod, layout, group):
    n, k, m = 1000, 1024, 5
    rng = np.random.Generator(np.random.Philox(key=[5, group]))
    weights, _ = _tensor(qx, oracle_mod, rng, layout, group, n, k)
    clean = rng.standard_normal((m, k)).astype(np.float32)
    x = clean.copy()
    x[1, 3], x[2, 700] = np.inf, np.nan
    for x_type in (BF16, F16):
        status, y = weights.qgemm_storage(_storage(x, x_type)[0], x_type, m)
        assert status == qx.OK and not np.isfinite(y[1]).any() and np.isnan(y[2]).all()
        status, want = weights.qgemm_storage(_storage(clean, x_type)[0], x_type, m)
        assert status == qx.OK and np.array_equal(y[[0, 3, 4]].view(np.uint32), want[[0, 3, 4]].view(np.uint32))


# back to back on one scratch, with nothing waiting between: each call's activations take the place of those that the
# call in front may still be reading, and the launches overlap
@pytest.mark.parametrize("layout,group,m,x_type", [(INT8, 0, 3, BF16), (UINT4, 128, 12, F16), (UINT4, 128, 6, F32)])
def test_chained_calls(qx, oracle_mod, layout, group, m, x_type):
    import torch
    n, k = 4096, 4096
    rng = np.random.Generator(np.random.Philox(key=[9, group + m]))
    weights, _ = _tensor(qx, oracle_mod, rng, layout, group, n, k)
    types = {F32: torch.float32, F16: torch.float16, BF16: torch.bfloat16}
    xs = [torch.randn((m, k), device="cuda").to(types[x_type]) for _ in range(3)]
    want = []
    for x in xs:
        want.append(torch.zeros((m, n), device="cuda"))
        assert weights.qgemm_storage_dev(x, x_type, want[-1], F32, m) == qx.OK, qx.last_error()
        torch.cuda.synchronize()
    got = [torch.zeros((m, n), device="cuda") for _ in range(60)]
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        assert weights.qgemm_storage_dev(xs[i % 3], x_type, y, F32, m) == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i % 3]) for i, y in enumerate(got))


def test_chained_w4a8(qx):
    import torch
    m, n, k = 16, 4096, 4096
    w = torch.randint(0, 256, (n * k // 2,), dtype=torch.uint8, device="cuda")
    ws = torch.rand(n, device="cuda") + 0.5
    scratch = torch.zeros(int(qx.lib.qx_lowbit_w8a8_scratch_bytes(m, k)), dtype=torch.uint8, device="cuda")
    xs = [torch.randn((m, k), device="cuda") for _ in range(3)]

    def call(x, y):
        assert qx.lib.qx_lowbit_gemm_w8a8_dev(w.data_ptr(), ws.data_ptr(), x.data_ptr(), y.data_ptr(), scratch.data_ptr(),
                                              m, n, k, torch.cuda.current_stream().cuda_stream) == qx.OK, qx.last_error()

    want = [torch.zeros((m, n), device="cuda") for _ in xs]
    for x, y in zip(xs, want):
        call(x, y)
        torch.cuda.synchronize()
    got = [torch.zeros((m, n), device="cuda") for _ in range(60)]
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        call(xs[i % 3], y)
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i % 3]) for i, y in enumerate(got))
