"""How far f32 results of batched projections are from float64: the 2-norm of the difference over that of
the result, in the place of a bound per element, which is too wide to show a few more roundings."""

import numpy as np
import pytest

from test_canonical_gpu import BF16, F16, F32, INT4, INT8, UINT4

pytestmark = pytest.mark.gpu

GROUP, CHANNEL = 4, 3
TYPES = {F32: "float32", F16: "float16", BF16: "bfloat16"}


def canonical_error(qx, layout, group, m, n, k, x_type, seed=3):
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
    assert weights.qgemm_storage_dev(x, x_type, y, F32, m) == qx.OK, qx.last_error()
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
    return ((y.double() - exact).norm() / exact.norm()).item()


# exact sums of the whole row: what is left are the roundings of four partial sums and of the two
# factors, together less than one 2^-24 of the result
@pytest.mark.parametrize("m,n,k,x_type", [(1024, 2048, 2048, F16), (1024, 2048, 2048, BF16), (300, 4096, 4096, F16)])
def test_row_scaled_int8(qx, m, n, k, x_type):
    assert canonical_error(qx, INT8, 0, m, n, k, x_type) <= 2.0 ** -24
