"""Calls on host buffers give the bits of the device entry point, whichever way the operands take: pinned memory,
pageable memory up to the size that passes through the library's own pinned memory, and beyond."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 65536 floats is the line: activations at it and above, results at it and above; and activations off 16 bytes
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("m,n,k,offset", [(1, 256, 256, 0), (1, 300, 1024, 1), (32, 128, 2048, 0), (32, 130, 2080, 0),
                                          (32, 2048, 256, 0), (32, 2049, 256, 2)])
def test_host_equals_device(qx, wl, pinned, m, n, k, offset):
    import torch
    weights = qx.PackedWeights()
    assert weights.prepare(0, wl.packed_blocks(0, n, k, 0.001, 0.02, seed=n), n, k) == qx.OK, qx.last_error()
    for seed in (1, 2):  # (the second call reuses the memory)
        x = torch.zeros(m * k + offset, pin_memory=pinned)[offset:]
        x[:] = torch.from_numpy(wl.activations_f32(m, k, seed=seed).reshape(-1))
        y = torch.full((m, n), float("nan"), pin_memory=pinned)
        status, got = weights.qgemm_prepacked(x.numpy(), m, y.numpy())
        assert status == qx.OK, qx.last_error()
        want = torch.zeros((m, n), device="cuda")
        assert weights.qgemm_dev(x.cuda().view(m, k), want, m) == qx.OK, qx.last_error()
        assert np.array_equal(got.view(np.uint32), want.cpu().numpy().view(np.uint32))


# Buffers that are on the device already (the copies of a host call have always taken them), below and above the size
# that passes through pinned memory: the CPU must not touch them
@pytest.mark.parametrize("m,n,k", [(1, 256, 256), (2, 4096, 1024), (32, 4096, 2080)])
def test_device_buffers_in_a_host_call(qx, wl, m, n, k):
    import torch
    weights = qx.PackedWeights()
    assert weights.prepare(0, wl.packed_blocks(0, n, k, 0.001, 0.02, seed=n), n, k) == qx.OK, qx.last_error()
    x = torch.from_numpy(wl.activations_f32(m, k, seed=3)).view(m, k)
    want = torch.zeros((m, n), device="cuda")
    assert weights.qgemm_dev(x.cuda(), want, m) == qx.OK, qx.last_error()
    for x_device, y_device in ((True, False), (False, True), (True, True)):
        xs, y = x.cuda() if x_device else x, torch.full((m, n), float("nan"), device="cuda" if y_device else "cpu")
        torch.cuda.synchronize()  # (the call runs on a stream of its own)
        assert weights.qgemm_prepacked_ptr(xs.data_ptr(), y.data_ptr(), m) == qx.OK, qx.last_error()
        assert torch.equal(y.cuda(), want)
