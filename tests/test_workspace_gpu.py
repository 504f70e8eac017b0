"""A workspace that has served the largest batch serves every smaller one without growing, whatever route
that takes, so smaller batches may be captured; and calls that share one in turn, or run beside each other
on two streams with one each, do not disturb each other."""

import ctypes as C

import numpy as np
import pytest

from test_canonical_gpu import BF16, F16, F32, INT4, INT8, UINT4
from test_scaled_gemm_gpu import _tensor

pytestmark = pytest.mark.gpu

TORCH = {F32: "float32", F16: "float16", BF16: "bfloat16"}


class Workspace:
    def __init__(self, qx):
        self.qx, self.handle = qx, C.c_void_p()
        assert qx.lib.qx_workspace_create(0, C.byref(self.handle)) == qx.OK, qx.last_error()

    def capacity(self):
        return self.qx.lib.qx_workspace_capacity(self.handle)

    def close(self):
        self.qx.lib.qx_workspace_destroy(self.handle)


def canonical_call(qx, weights, x, x_type, y, workspace):
    import torch
    return qx.lib.qx_qgemm_prepacked_epilogue_storage_dev(
        weights.handle, C.c_void_p(x.data_ptr()), x_type, None, C.c_void_p(y.data_ptr()), F32, x.shape[0], 0,
        workspace.handle, C.c_void_p(torch.cuda.current_stream().cuda_stream))


def panel_call(qx, weights, x, y, workspace):
    import torch
    return qx.lib.qx_qgemm_prepacked_bf16_dev(
        weights.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), x.shape[0], y.shape[1], workspace.handle,
        C.c_void_p(torch.cuda.current_stream().cuda_stream))


def captured(qx, call):
    """`call` in a graph of its own, replayed once."""
    import torch
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        status = call()
    assert status == qx.OK, qx.last_error()
    graph.replay()
    torch.cuda.synchronize()


# (4736 rows are 37 weight tiles: 512 tokens fill 148 SMs with whole tiles, smaller batches are cut)
@pytest.mark.parametrize("act_order", [False, True])
def test_smaller_canonical_batches_are_captured(qx, oracle_mod, act_order):
    import torch
    n, k = 4736, 1024
    rng = np.random.Generator(np.random.Philox(key=[1, int(act_order)]))
    order = rng.permutation(k).astype(np.int32) if act_order else None
    weights, _ = _tensor(qx, oracle_mod, rng, UINT4, 128, n, k, act_order=order)
    workspace = Workspace(qx)
    x = torch.randn((512, k), device="cuda").bfloat16()
    y = torch.zeros((512, n), device="cuda")
    assert canonical_call(qx, weights, x, BF16, y, workspace) == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    capacity = workspace.capacity()
    for m, x_type in [(300, F32), (129, BF16), (128, F16), (100, BF16), (64, F32), (33, BF16), (16, F16), (5, BF16), (1, F32)]:
        xs = torch.randn((m, k), device="cuda").to(getattr(torch, TORCH[x_type]))
        got, want = torch.zeros((m, n), device="cuda"), torch.zeros((m, n), device="cuda")
        captured(qx, lambda: canonical_call(qx, weights, xs, x_type, got, workspace))
        assert workspace.capacity() == capacity
        assert weights.qgemm_storage_dev(xs, x_type, want, F32, m) == qx.OK, qx.last_error()
        torch.cuda.synchronize()
        assert torch.equal(got, want), (m, x_type)
    workspace.close()


# Batches that stream their codes, on a workspace of their own: smaller ones of any type, off 16 bytes as well, take digit
# images, digit planes, laid-out activations or the tensor cores
@pytest.mark.parametrize("layout,group,n,k,order,m,x_type,smaller", [
    (UINT4, 128, 4736, 1024, False, 8, BF16, [(8, F32), (5, F16), (4, BF16), (1, F32)]),
    (UINT4, 128, 4736, 1024, False, 16, F16, [(16, F32), (9, BF16), (8, F16), (4, F32)]),
    (INT4, 32, 4096, 2048, True, 6, F16, [(6, F32), (4, BF16), (1, F32)]),
    (INT4, 128, 64, 40960, True, 5, BF16, [(5, F32), (4, F32), (1, F16)]),
    (UINT4, 128, 8192, 8192, False, 32, F16, [(32, F32), (25, F32), (24, F32), (16, BF16), (1, F32)]),
    (INT8, 0, 16384, 32, False, 8, BF16, [(7, F32), (5, BF16), (4, F32), (1, F16)]),
    (INT8, 0, 4096, 4096, False, 16, BF16, [(12, F32), (8, F16), (5, BF16), (4, F32), (1, BF16)]),
    (INT8, 0, 32, 40000, False, 4, F32, [(3, F32), (1, BF16)]),
])
def test_smaller_batches_of_a_streamed_one_are_captured(qx, oracle_mod, layout, group, n, k, order, m, x_type, smaller):
    import torch
    rng = np.random.Generator(np.random.Philox(key=[n + m, k]))
    weights, _ = _tensor(qx, oracle_mod, rng, layout, group, n, k,
                         act_order=rng.permutation(k).astype(np.int32) if order else None)
    workspace = Workspace(qx)
    x = torch.randn((m, k), device="cuda").to(getattr(torch, TORCH[x_type]))
    y = torch.zeros((m, n), device="cuda")
    assert canonical_call(qx, weights, x, x_type, y, workspace) == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    capacity = workspace.capacity()
    calls = []
    for rows, kind in smaller:
        for offset in (0, 1):
            buffer = torch.zeros(rows * k + 1, device="cuda", dtype=getattr(torch, TORCH[kind]))
            xs = buffer[offset:offset + rows * k].view(rows, k)
            xs.copy_(torch.randn((rows, k), device="cuda"))
            want = torch.zeros((rows, n), device="cuda")
            assert canonical_call(qx, weights, xs, kind, want, workspace) == qx.OK, qx.last_error()
            torch.cuda.synchronize()
            assert workspace.capacity() == capacity, (rows, kind, offset)
            calls.append((xs, kind, want))
    for xs, kind, want in calls:  # (nothing has grown: now inside a capture)
        got = torch.zeros_like(want)
        captured(qx, lambda: canonical_call(qx, weights, xs, kind, got, workspace))
        assert workspace.capacity() == capacity and torch.equal(got, want)
    workspace.close()


def test_smaller_q8_0_prompts_are_captured(qx, wl):
    import torch
    n, k = 4736, 1024
    weights = qx.PackedWeights()
    assert weights.prepare(0, wl.packed_blocks(0, n, k, 0.001, 0.02, seed=4), n, k) == qx.OK, qx.last_error()
    workspace = Workspace(qx)
    x = torch.randn((512, k), device="cuda").bfloat16()
    y = torch.zeros((512, n), device="cuda")
    assert panel_call(qx, weights, x, y, workspace) == qx.OK, qx.last_error()
    torch.cuda.synchronize()
    capacity = workspace.capacity()
    for m in (400, 128, 65, 64, 17, 16, 8, 1):
        got, want = torch.zeros((m, n), device="cuda"), torch.zeros((m, n), device="cuda")
        captured(qx, lambda: panel_call(qx, weights, x[:m], got, workspace))
        assert workspace.capacity() == capacity
        assert weights.qgemm_bf16_dev(x[:m].view(torch.int16), want, m) == qx.OK, qx.last_error()
        torch.cuda.synchronize()
        assert torch.equal(got, want), m
    workspace.close()


def test_routes_in_turn_and_two_streams(qx, oracle_mod):
    import torch
    rng = np.random.Generator(np.random.Philox(key=[7, 8]))
    jobs = []
    for layout, group, n, k, m, x_type in [(UINT4, 128, 4096, 2048, 100, BF16), (INT8, 0, 2048, 2048, 40, BF16),
                                           (INT4, 32, 4096, 1024, 64, F16), (UINT4, 128, 4096, 2048, 1, F32)]:
        weights, _ = _tensor(qx, oracle_mod, rng, layout, group, n, k)
        x = torch.randn((m, k), device="cuda").to(getattr(torch, TORCH[x_type]))
        want = torch.zeros((m, n), device="cuda")
        assert weights.qgemm_storage_dev(x, x_type, want, F32, m) == qx.OK, qx.last_error()
        jobs.append((weights, x, x_type, want))
    torch.cuda.synchronize()
    streams, workspaces = [torch.cuda.Stream() for _ in range(2)], [Workspace(qx) for _ in range(2)]
    results = []
    for round_ in range(6):
        for side in range(2):
            with torch.cuda.stream(streams[side]):
                for i in range(len(jobs)):
                    weights, x, x_type, want = jobs[(i + side) % len(jobs)]
                    y = torch.zeros_like(want)
                    assert canonical_call(qx, weights, x, x_type, y, workspaces[side]) == qx.OK, qx.last_error()
                    results.append((y, want))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want) for y, want in results)
    assert qx.lib.qx_check_device_errors() == qx.OK, qx.last_error()
    for workspace in workspaces:
        workspace.close()
