"""How far f32 results of batched projections are from float64: the 2-norm of the difference over that of
the result, in the place of a bound per element, which is too wide to show a few more roundings."""

import numpy as np
import pytest

from test_canonical_gpu import BF16, F16, F32, INT4, INT8, UINT4

pytestmark = pytest.mark.gpu

GROUP, CHANNEL = 4, 3
TYPES = {F32: "float32", F16: "float16", BF16: "bfloat16"}


def relative(y, exact):
    return ((y.double() - exact).norm() / exact.norm()).item()


def canonical_error(qx, layout, group, m, n, k, x_type, batch=None, seed=3):
    """Error of all m tokens, computed `batch` at a time (None: in one call)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    groups = k // group if group else 1
    scales = torch.rand(n * groups, generator=g, device="cuda") * 0.01 + 0.005
    data = torch.randint(0, 256, (n * k // (1 if layout == INT8 else 2),), generator=g, device="cuda", dtype=torch.uint8)
    zeros = torch.randint(0, 16, (n * groups,), generator=g, device="cuda").float() if layout == UINT4 else None
    host = [None if a is None else a.cpu().numpy() for a in (data, scales, zeros)]
    weights = qx.CanonicalWeights()
    view = qx.canonical_view(layout, GROUP if group else CHANNEL, n, k, group or k, host[0], host[1], zeros=host[2])
    assert weights.prepare(view) == qx.OK, qx.last_error()
    x = torch.randn((m, k), generator=g, device="cuda").to(getattr(torch, TYPES[x_type]))
    y = torch.zeros((m, n), device="cuda")
    for first in range(0, m, batch or m):
        rows = slice(first, min(m, first + (batch or m)))
        assert weights.qgemm_storage_dev(x[rows], x_type, y[rows], F32, rows.stop - rows.start) == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    if layout == INT8:
        q = data.view(torch.int8).double()
    else:
        q = torch.stack((data & 15, data >> 4), dim=-1).view(-1).double()
        if layout == INT4:
            q = torch.where(q >= 8, q - 16, q)
    q = q.view(n, groups, -1)
    if zeros is not None:
        q = q - zeros.double().view(n, groups, 1)
    exact = x.double() @ (q * scales.double().view(n, groups, 1)).view(n, k).T
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()
    return relative(y, exact)


# exact sums of the whole row: what is left are the roundings of four partial sums and of the two
# factors, together less than one 2^-24 of the result
@pytest.mark.parametrize("m,n,k,x_type", [(1024, 2048, 2048, F16), (1024, 2048, 2048, BF16), (300, 4096, 4096, F16)])
def test_row_scaled_int8(qx, m, n, k, x_type):
    assert canonical_error(qx, INT8, 0, m, n, k, x_type) <= 2.0 ** -24


# Batches on the tensor cores against the digit kernels, which up to four tokens take: same values,
# exact sums of 16 columns
@pytest.mark.parametrize("layout,group,m,n,k,x_type", [
    (UINT4, 32, 64, 2048, 4096, BF16), (UINT4, 128, 128, 1024, 4096, F16), (INT4, 32, 512, 1024, 8192, BF16),
    (INT4, 64, 16, 2048, 2048, F16), (INT8, 128, 64, 2048, 4096, F16), (INT8, 64, 100, 2048, 1024, BF16),
    (UINT4, 128, 64, 2048, 4096, F32), (INT8, 128, 32, 2048, 4096, F32)])
def test_batches_no_further_than_single_tokens(qx, layout, group, m, n, k, x_type):
    assert canonical_error(qx, layout, group, m, n, k, x_type) <= canonical_error(qx, layout, group, m, n, k, x_type, 4)


# q8_0 prompts against the decode kernels on the widened activations
@pytest.mark.parametrize("m,n,k", [(331, 4096, 1024), (64, 2048, 2048), (128, 2048, 4096), (40, 1024, 8192), (331, 1024, 11008)])
def test_q8_0_prompts_no_further_than_the_decode_kernels(qx, wl, m, n, k):
    import torch
    packed = wl.packed_blocks(0, n, k, 0.001, 0.02, seed=n + k)
    blocks = torch.from_numpy(packed).cuda().view(n, k // 32, 34)
    w = (blocks[..., :2].contiguous().view(torch.float16).double() * blocks[..., 2:].contiguous().view(torch.int8).double()).view(n, k)
    weights = qx.PackedWeights()
    assert weights.prepare(0, packed, n, k) == qx.OK, qx.last_error()
    x = torch.randn((m, k), generator=torch.Generator(device="cuda").manual_seed(m), device="cuda").bfloat16()
    y, y_decode = torch.zeros((m, n), device="cuda"), torch.zeros((m, n), device="cuda")
    assert weights.qgemm_bf16_dev(x.view(torch.int16), y, m) == qx.OK, qx.last_error()
    assert weights.qgemm_dev(x.float(), y_decode, m) == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    exact = x.double() @ w.T
    assert relative(y, exact) <= relative(y_decode, exact)
